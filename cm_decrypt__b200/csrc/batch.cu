// Host side of the fused path: round lists for single-key and mixed batches,
// the persistent-grid sizing, and the pinned staging buffer.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "engine.h"

namespace cmd {

int fused_blocks_per_sm(int single_set, int wpb, size_t smem);

int HostScratch::reserve(size_t bytes)
{
    if (bytes <= cap)
        return CMD_OK;
    if (ptr)
        cudaFreeHost(ptr);
    ptr = nullptr;
    cap = 0;
    cudaError_t e = cudaMallocHost(&ptr, bytes);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaMallocHost");
    cap = bytes;
    return CMD_OK;
}

void HostScratch::release()
{
    if (ptr)
        cudaFreeHost(ptr);
    ptr = nullptr;
    cap = 0;
}

int TileCounter::begin(cmd_engine *eng, cudaStream_t s)
{
    cudaError_t e = cudaSuccess;
    if (capturing(s)) {
        constexpr unsigned BLOCK = 256;
        if (eng->graph_counters_left == 0) {
            BesideCapture beside;
            void *p = nullptr;
            e = cudaMalloc(&p, BLOCK * 4);
            if (e != cudaSuccess)
                return cuda_fail(e, "cudaMalloc(counters)");
            eng->graph_counters.push_back(static_cast<uint32_t *>(p));
            eng->graph_counters_left = BLOCK;
        }
        ptr = eng->graph_counters.back() + --eng->graph_counters_left;
        return CMD_OK;
    }
    const unsigned i = eng->counter_next++ % COUNTER_RING;
    if (!eng->counter_done[i])
        e = cudaEventCreateWithFlags(&eng->counter_done[i], cudaEventDisableTiming);
    else
        e = cudaStreamWaitEvent(s, eng->counter_done[i]);
    ptr = eng->tile_counter + COUNTER_RING0 + i;
    done = eng->counter_done[i];
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "work counter");
}

int TileCounter::end(cudaStream_t s, int rc)
{
    const cudaError_t e = done ? cudaEventRecord(done, s) : cudaSuccess;
    return rc ? rc : e == cudaSuccess ? CMD_OK : cuda_fail(e, "work counter");
}

// Persistent grid: resident CTAs per SM (occupancy with this smem) x SMs,
// never more CTAs than rounds.
static int grid_for(cmd_engine *eng, int single_set, int wpb, size_t smem, uint64_t rounds)
{
    int per_sm = fused_blocks_per_sm(single_set, wpb, smem);
    if (per_sm < 1)
        per_sm = 1;
    uint64_t g = (uint64_t)per_sm * (uint64_t)eng->num_sms;
    return (int)std::min<uint64_t>(g, rounds);
}

// Ciphertexts per round.  `full` (every round fills all WPB warps) leaves
// the last wave partly idle when the batch is not a multiple of the resident
// capacity; `balanced` shrinks rounds (in whole 32-ciphertext tiles) so the
// batch splits into equal shares per resident CTA.
static uint32_t round_size(cmd_engine *eng, int set, int wpb, size_t count, bool balanced)
{
    const uint64_t full = (uint64_t)wpb * 32;
    if (!balanced)
        return (uint32_t)full;
    int per_sm = fused_blocks_per_sm(set, wpb, fused_smem(set, wpb));
    const uint64_t ctas = (uint64_t)(per_sm < 1 ? 1 : per_sm) * eng->num_sms;
    const uint64_t waves = (count + ctas * full - 1) / (ctas * full);
    uint64_t r = (count + ctas * waves - 1) / (ctas * waves);
    r = (r + 31) / 32 * 32;
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(r, 32), full);
}

uint32_t fused_round(cmd_engine *eng, int set, size_t count)
{
    return round_size(eng, set, eng->fcfg[set].wpb, count, eng->fcfg[set].balanced);
}

int run_fused_counter(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                      uint16_t *d_weight, cudaStream_t s, uint32_t *counter, uint16_t *d_pos, int balanced,
                      uint32_t round_cts, uint8_t *err_packed)
{
    const int set = key->dev.set;
    const SetInfo si = set_info(set);
    const int wpb = eng->fcfg[set].wpb;
    if (round_cts % 32 != 0 || round_cts > (uint32_t)wpb * 32) {
        set_last_error("fused round of " + std::to_string(round_cts) +
                       " ciphertexts: must be a multiple of 32 and at most " + std::to_string(wpb * 32));
        return CMD_E_ARG;
    }
    const uint32_t round = round_cts ? round_cts
                                     : round_size(eng, set, wpb, count,
                                                  balanced < 0 ? eng->fcfg[set].balanced : balanced != 0);
    const uint64_t rounds = (count + round - 1) / round;
    if (rounds > 0xFFFFFFFFull) {
        set_last_error("batch needs more than 2^32 fused rounds");
        return CMD_E_ARG;
    }
    FusedArgs a;
    memset(&a, 0, sizeof a);
    a.tiles = nullptr;
    a.ntiles = (uint32_t)rounds;
    a.round_cts = round;
    a.total = count;
    a.keys = nullptr;
    a.key0 = key_ref(key->dev);
    a.cts = d_cts;
    a.err = d_err;
    a.weight = d_weight;
    a.tile_counter = counter;
    a.single_set = set;
    fill_fft(a, eng);
    a.err_stride = (uint32_t)si.nw;
    a.pos = d_pos;
    a.pos_stride = (uint32_t)(si.t + 1);
    a.err_packed = err_packed;
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaMemsetAsync(counter)");
    const int grid = grid_for(eng, set, wpb, fused_smem(set, wpb), rounds);
    e = launch_fused(a, grid, wpb, s, LaunchCounter{&eng->launches});
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "fused kernel launch");
}

// Sets the fused kernel's shared-memory attribute for this set's current
// configuration ahead of time (e.g. before a stream capture begins).
cudaError_t fused_prepare(cmd_engine *eng, int set)
{
    const int wpb = eng->fcfg[set].wpb;
    return fused_blocks_per_sm(set, wpb, fused_smem(set, wpb)) > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
}

int run_fused_single(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                     uint16_t *d_weight, cudaStream_t s, uint16_t *d_pos)
{
    TileCounter counter;
    const int rc = counter.begin(eng, s);
    return rc ? rc : counter.end(s, run_fused_counter(eng, key, d_cts, count, d_err, d_weight, s, counter.ptr, d_pos, -1));
}

// Set shared by every ciphertext of a mixed batch, or -1.
int mixed_single_set(const int *key_set, const uint32_t *key_idx, size_t count)
{
    if (count == 0)
        return -1;
    const int s0 = key_set[key_idx[0]];
    for (size_t c = 1; c < count; c++)
        if (key_set[key_idx[c]] != s0)
            return -1;
    return s0;
}

// Groups ciphertexts by key (counting sort, stable in batch order) into
// `order` and cuts each key's run into rounds of up to R; rounds of costlier
// sets come first so the dynamic scheduler ends with cheap rounds.
void plan_mixed(const int *key_set, size_t nkeys, const uint32_t *key_idx, size_t count, uint32_t R,
                std::vector<uint32_t> &order, std::vector<FusedTile> &tiles)
{
    std::vector<uint32_t> cnt(nkeys + 1, 0);
    for (size_t c = 0; c < count; c++)
        cnt[key_idx[c] + 1]++;
    for (size_t k = 0; k < nkeys; k++)
        cnt[k + 1] += cnt[k];
    order.assign(count, 0);
    std::vector<uint32_t> fill(cnt.begin(), cnt.end() - 1);
    for (size_t c = 0; c < count; c++)
        order[fill[key_idx[c]]++] = (uint32_t)c;
    tiles.clear();
    for (size_t k = 0; k < nkeys; k++)
        for (uint32_t r0 = cnt[k]; r0 < cnt[k + 1]; r0 += R)
            tiles.push_back(FusedTile{(uint32_t)k, std::min(R, cnt[k + 1] - r0), r0});
    auto cost = [&](const FusedTile &t) {
        const SetInfo si = set_info(key_set[t.key]);
        return (uint64_t)si.n * si.t * si.m * si.m;
    };
    std::stable_sort(tiles.begin(), tiles.end(),
                     [&](const FusedTile &x, const FusedTile &y) { return cost(x) > cost(y); });
}

// A mixed batch on the staged kernels, set by set: slots grouped by key, each key's
// run cut into tiles and syndrome blocks; passes of at most as many tiles as the
// parts of a single-key batch in flight, since every key's last tile takes the scratch
// of a full one (46 KB), however few ciphertexts it has.
struct StagedSlice {
    int set, pass;
    uint32_t block0, nblocks, tile0, ntiles;
};
struct StagedPlan {
    std::vector<uint32_t> order;
    std::vector<StagedPiece> blocks, tiles;
    std::vector<StagedSlice> slices;  // by pass, the costlier sets first
};
constexpr uint32_t STAGED_PASS_TILES = STAGED_STREAMS * 65536 / 32;

static void plan_staged(const int *key_set, size_t nkeys, const uint32_t *key_idx, size_t count, StagedPlan &p)
{
    std::vector<uint32_t> cnt(nkeys + 1, 0);
    for (size_t c = 0; c < count; c++)
        cnt[key_idx[c] + 1]++;
    for (size_t k = 0; k < nkeys; k++)
        cnt[k + 1] += cnt[k];
    p.order.resize(count);
    std::vector<uint32_t> fill(cnt.begin(), cnt.end() - 1);
    for (size_t c = 0; c < count; c++)
        p.order[fill[key_idx[c]]++] = (uint32_t)c;
    constexpr uint32_t bs = 32 * staged_block_tiles;
    uint32_t room = STAGED_PASS_TILES;  // tiles left in the pass
    int pass = 0;
    for (int st = NSETS - 1; st >= 0; st--) {
        for (size_t k = 0; k < nkeys; k++) {
            if (key_set[k] != st)
                continue;
            for (uint32_t r = cnt[k]; r < cnt[k + 1]; r += bs) {
                const uint32_t n = std::min(cnt[k + 1] - r, bs), nt = (n + 31) / 32;
                if (nt > room) {
                    pass++;
                    room = STAGED_PASS_TILES;
                }
                if (p.slices.empty() || p.slices.back().set != st || p.slices.back().pass != pass)
                    p.slices.push_back(StagedSlice{st, pass, (uint32_t)p.blocks.size(), 0, (uint32_t)p.tiles.size(), 0});
                StagedSlice &sl = p.slices.back();
                p.blocks.push_back(StagedPiece{(uint32_t)k, n, r, sl.ntiles});
                for (uint32_t i = 0; i < n; i += 32)
                    p.tiles.push_back(StagedPiece{(uint32_t)k, std::min(n - i, 32u), r + i, 0});
                sl.nblocks++;
                sl.ntiles += nt;
                room -= nt;
            }
        }
    }
}

static size_t al256(size_t x) { return (x + 255) / 256 * 256; }

// CMD_E_BUDGET: nothing ran, the fused kernel has to.  Caller holds eng->mu.
static int run_mixed_staged(cmd_engine *eng, const cmd_key *const *keys, size_t nkeys, const int *key_set,
                            const uint32_t *h_key_idx, const uint8_t *d_cts, const uint64_t *h_ct_off, size_t count,
                            uint32_t *d_err, const uint64_t *h_err_off, uint16_t *d_weight, cudaStream_t s)
{
    StagedPlan p;
    plan_staged(key_set, nkeys, h_key_idx, count, p);
    std::vector<FusedKeyRef> krefs(nkeys);
    for (size_t k = 0; k < nkeys; k++)
        krefs[k] = key_ref(keys[k]->dev);
    const size_t b_order = al256(count * 4), b_off = al256(count * 8), b_blk = al256(p.blocks.size() * sizeof(StagedPiece)),
                 b_tile = al256(p.tiles.size() * sizeof(StagedPiece)), b_keys = al256(nkeys * sizeof(FusedKeyRef));
    size_t words = 0, at_word = 0;  // of the largest pass; of a pass so far
    for (size_t i = 0; i < p.slices.size(); i++) {
        if (i == 0 || p.slices[i].pass != p.slices[i - 1].pass)
            at_word = 0;
        at_word += staged_scratch_words(p.slices[i].set, 32 * (size_t)p.slices[i].ntiles);
        words = std::max(words, at_word);
    }
    int rc = eng->staged.reserve(eng, words * 4, CMD_E_BUDGET);
    if (rc)
        return rc;
    if (eng->fused.begin(eng, b_order + 2 * b_off + b_blk + b_tile + b_keys, s) != CMD_OK)
        return CMD_E_BUDGET;
    uint8_t *at = static_cast<uint8_t *>(eng->fused.ptr);
    cudaError_t e = cudaSuccess;
    auto put = [&](const void *src, size_t bytes, size_t room) {
        uint8_t *dst = at;
        at += room;
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
        return dst;
    };
    StagedMixed mx;
    mx.order = reinterpret_cast<const uint32_t *>(put(p.order.data(), count * 4, b_order));
    mx.ct_off = reinterpret_cast<const uint64_t *>(put(h_ct_off, count * 8, b_off));
    mx.err_off = reinterpret_cast<const uint64_t *>(put(h_err_off, count * 8, b_off));
    mx.blocks = reinterpret_cast<const StagedPiece *>(put(p.blocks.data(), p.blocks.size() * sizeof(StagedPiece), b_blk));
    mx.tiles = reinterpret_cast<const StagedPiece *>(put(p.tiles.data(), p.tiles.size() * sizeof(StagedPiece), b_tile));
    mx.keys = reinterpret_cast<const FusedKeyRef *>(put(krefs.data(), nkeys * sizeof(FusedKeyRef), b_keys));
    if (e != cudaSuccess)
        return eng->fused.end(s, e);
    // the sets of a pass beside one another, as the parts of a single-key batch
    const int ns = STAGED_STREAMS;
    for (size_t i = 0; i < p.slices.size() && rc == CMD_OK;) {
        if ((rc = staged_begin(eng, words * 4, ns, s)))
            break;
        const int pass = p.slices[i].pass;
        uint32_t *scratch = static_cast<uint32_t *>(eng->staged.ptr);
        for (int k = 0; i < p.slices.size() && p.slices[i].pass == pass && e == cudaSuccess; i++, k++) {
            const StagedSlice &sl = p.slices[i];
            StagedMixed m = mx;
            m.blocks += sl.block0;
            m.tiles += sl.tile0;
            e = launch_staged_mixed(sl.set, m, sl.nblocks, sl.ntiles, d_cts, scratch, d_err, d_weight, eng->fft[sl.set],
                                    eng->num_sms, eng->piece_stream[k % ns], LaunchCounter{&eng->launches});
            scratch += staged_scratch_words(sl.set, 32 * (size_t)sl.ntiles);
        }
        rc = staged_end(eng, ns, s, e);
    }
    const int r = eng->fused.end(s);
    return rc ? rc : r;
}

// A small mixed batch on the per-ciphertext kernels.  CMD_E_BUDGET as above, also
// when an offset does not fit an item.
static int run_mixed_small(cmd_engine *eng, const cmd_key *const *keys, const uint32_t *h_key_idx, const uint8_t *d_cts,
                           const uint64_t *h_ct_off, size_t count, uint32_t *d_err, const uint64_t *h_err_off,
                           uint16_t *d_weight, cudaStream_t s)
{
    std::vector<LatItem> items(count);
    for (size_t c = 0; c < count; c++) {
        if ((h_ct_off[c] | h_err_off[c]) >> 32)
            return CMD_E_BUDGET;
        const KeyDev &k = keys[h_key_idx[c]]->dev;
        items[c] = LatItem{k.wfft, k.bctl, (uint32_t)h_ct_off[c], (uint32_t)h_err_off[c], k.set, 0, nullptr};
    }
    const size_t b_items = al256(count * sizeof(LatItem)), b_mid = count > CT_ONE_LAUNCH ? count * 512 : 0;
    int rc = staged_begin(eng, b_items + b_mid, 1, s);
    if (rc)
        return rc;
    uint8_t *base = static_cast<uint8_t *>(eng->staged.ptr);
    cudaError_t e = cudaMemcpyAsync(base, items.data(), count * sizeof(LatItem), cudaMemcpyHostToDevice, s);
    FftPlans plans;
    for (int st = 0; st < NSETS; st++)
        plans.p[st] = eng->fft[st];
    if (e == cudaSuccess)
        e = launch_ct_items(reinterpret_cast<const LatItem *>(base), d_cts, (uint32_t)count, (uint32_t)count,
                            reinterpret_cast<uint16_t *>(base + b_items), d_err, d_weight, nullptr, plans, eng->num_sms,
                            s, LaunchCounter{&eng->launches});
    return staged_end(eng, 1, s, e);
}

int fused_grid(cmd_engine *eng, int single_set, int wpb, size_t smem, uint64_t rounds)
{
    return grid_for(eng, single_set, wpb, smem, rounds);
}

}  // namespace cmd

using namespace cmd;

extern "C" int cmd_decrypt_mixed_device(cmd_engine *eng, const cmd_key *const *keys, size_t nkeys,
                                        const uint32_t *h_key_idx, const uint8_t *d_cts, const uint64_t *h_ct_off,
                                        size_t count, uint32_t *d_err, const uint64_t *h_err_off,
                                        uint16_t *d_weight, void *stream)
{
    if (!eng || (count && (!keys || !nkeys || !h_key_idx || !d_cts || !h_ct_off || !d_err || !h_err_off)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    if (count > 0xFFFFFFFFull || nkeys > 0xFFFFFFFFull) {
        set_last_error("mixed batch: more than 2^32 ciphertexts or keys");
        return CMD_E_ARG;
    }
    for (size_t k = 0; k < nkeys; k++)
        if (!keys[k] || keys[k]->eng != eng) {
            set_last_error("mixed batch: key " + std::to_string(k) + " is null or belongs to another engine");
            return CMD_E_ARG;
        }
    cudaSetDevice(eng->device);
    cudaStream_t s = stream ? (cudaStream_t)stream : eng->stream;

    for (size_t c = 0; c < count; c++)
        if (h_key_idx[c] >= nkeys) {
            set_last_error("mixed batch: ciphertext " + std::to_string(c) + " names key " +
                           std::to_string(h_key_idx[c]) + " of " + std::to_string(nkeys));
            return CMD_E_ARG;
        }
    std::vector<int> kset(nkeys);
    for (size_t k = 0; k < nkeys; k++)
        kset[k] = keys[k]->dev.set;
    // As run_auto (engine.cu): per-ciphertext kernels up to 24 an SM, then the staged
    // ones; the fused kernel for about one round of its warps, when their scratch
    // does not fit and under stream capture.  64 keys on a B200, fused -> taken:
    // 300 ciphertexts 985 -> 145 us, 1,000 1,271 -> 231 us, 10,000 1,797 -> 1,272 us,
    // 20,000 1,843 -> 1,653 us, 100,000 4,088 -> 3,829 us; 40,000 1,910 us (staged
    // 2,023 us).  The staged kernels' cost is by tile and syndrome block, the fused
    // kernel's by round, a key has at least one of each, and a round costs more: 5,000
    // ciphertexts of 3,000 keys 11,557 -> 4,538 us, of as many keys 23,485 -> 8,491 us,
    // 28,000 of 1,000 keys 7,471 -> 2,996 us, 100,000 of 6,000 37,635 -> 11,691 us.
    std::lock_guard<std::mutex> lk(eng->mu);
    const size_t sms = (size_t)eng->num_sms;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!(count > 192 * sms && count <= 320 * sms) && cudaStreamIsCapturing(s, &cap) == cudaSuccess &&
        cap == cudaStreamCaptureStatusNone) {
        const int r = count <= CT_PER_SM * sms
                          ? run_mixed_small(eng, keys, h_key_idx, d_cts, h_ct_off, count, d_err, h_err_off, d_weight, s)
                          : run_mixed_staged(eng, keys, nkeys, kset.data(), h_key_idx, d_cts, h_ct_off, count, d_err,
                                             h_err_off, d_weight, s);
        if (r != CMD_E_BUDGET)
            return r;
    }
    cudaGetLastError();
    int single = mixed_single_set(kset.data(), h_key_idx, count);
    const int wpb = single >= 0 ? eng->fcfg[single].wpb : eng->fcfg_mixed.wpb;
    std::vector<uint32_t> order;
    std::vector<FusedTile> tiles;
    plan_mixed(kset.data(), nkeys, h_key_idx, count, (uint32_t)wpb * 32, order, tiles);
    std::vector<FusedKeyRef> krefs(nkeys);
    for (size_t k = 0; k < nkeys; k++)
        krefs[k] = key_ref(keys[k]->dev);

    // One device block for the work lists; pageable sources, so each copy has
    // consumed its host buffer when cudaMemcpyAsync returns.  Under capture the
    // graph's own block, filled now: a copy in the graph would read these vectors at
    // every replay.
    const size_t b_order = al256(count * 4), b_off = al256(count * 8), b_tiles = al256(tiles.size() * sizeof(FusedTile)),
                 b_keys = al256(nkeys * sizeof(FusedKeyRef)), need = b_order + 2 * b_off + b_tiles + b_keys;
    TileCounter counter;
    int rc = counter.begin(eng, s);
    if (rc)
        return rc;
    const bool graph = capturing(s);
    void *block = nullptr;
    cudaError_t e = cudaSuccess;
    uint32_t *d_order;
    uint64_t *d_ct_off, *d_err_off;
    FusedTile *d_tiles;
    FusedKeyRef *d_keys;
    {
        BesideCapture beside;
        if ((rc = graph ? graph_alloc(eng, need, &block) : eng->fused.begin(eng, need, s)))
            return counter.end(s, rc);
        uint8_t *at = static_cast<uint8_t *>(graph ? block : eng->fused.ptr);
        cudaStream_t up = graph ? eng->stream : s;
        auto put = [&]<class T>(T *&dst, const void *src, size_t bytes, size_t room) {
            dst = reinterpret_cast<T *>(at);
            at += room;
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, up);
        };
        put(d_order, order.data(), count * 4, b_order);
        put(d_ct_off, h_ct_off, count * 8, b_off);
        put(d_err_off, h_err_off, count * 8, b_off);
        put(d_tiles, tiles.data(), tiles.size() * sizeof(FusedTile), b_tiles);
        put(d_keys, krefs.data(), nkeys * sizeof(FusedKeyRef), b_keys);
        if (graph && e == cudaSuccess)
            e = cudaStreamSynchronize(up);
    }
    if (e == cudaSuccess)
        e = cudaMemsetAsync(counter.ptr, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess)
        return counter.end(s, eng->fused.end(s, e));
    FusedArgs a;
    memset(&a, 0, sizeof a);
    a.tiles = d_tiles;
    a.ntiles = (uint32_t)tiles.size();
    a.keys = d_keys;
    a.cts = d_cts;
    a.ct_off = d_ct_off;
    a.err_off = d_err_off;
    a.order = d_order;
    a.err = d_err;
    a.weight = d_weight;
    a.tile_counter = counter.ptr;
    a.single_set = single;
    fill_fft(a, eng);
    size_t smem = 0;
    if (single >= 0)
        smem = fused_smem(single, wpb);
    else
        for (int st = 0; st < NSETS; st++)
            smem = std::max(smem, fused_smem(st, wpb));
    const int grid = grid_for(eng, single, wpb, smem, tiles.size());
    e = launch_fused(a, grid, wpb, s, LaunchCounter{&eng->launches});
    return counter.end(s, eng->fused.end(s, e));
}

// C ABI of the decryption engine (include/cmd_b200.h): engine and key
// lifetime, the HBM budget, batch scheduling over the plain and fused kernel
// paths, and the host<->device staging for host-buffer calls.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "engine.h"

namespace cmd {
static int run_tile(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                    uint16_t *d_weight, uint16_t *d_pos, uint16_t *d_synd, cudaStream_t s, Scratch &buf);

static thread_local std::string g_last_error;
void set_last_error(const std::string &msg) { g_last_error = msg; }

int cuda_fail(cudaError_t e, const char *what)
{
    set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
    return CMD_E_CUDA;
}

bool valid_set(int set) { return set >= 0 && set < NSETS; }

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Charges `bytes` against the engine budget; false if it would not fit.
bool budget_take(cmd_engine *eng, size_t bytes)
{
    size_t cur = eng->used.load();
    while (true) {
        if (cur + bytes > eng->budget)
            return false;
        if (eng->used.compare_exchange_weak(cur, cur + bytes))
            return true;
    }
}
void budget_give(cmd_engine *eng, size_t bytes) { eng->used.fetch_sub(bytes); }

// Gives the staged scratch back; false if there is none.  Caller holds eng->mu, and
// reserves its own buffers before it begins on the staged scratch.
static bool give_back(cmd_engine *eng)
{
    if (!eng->staged.ptr)
        return false;
    eng->staged.release(eng);
    return true;
}

bool budget_take_first(cmd_engine *eng, size_t bytes)
{
    if (budget_take(eng, bytes))
        return true;
    std::lock_guard<std::mutex> lk(eng->mu);
    return give_back(eng) && budget_take(eng, bytes);
}

int device_alloc(cmd_engine *eng, void **p, size_t bytes, const char *what, const char *over)
{
    if (!budget_take_first(eng, bytes)) {
        set_last_error(over);
        return CMD_E_BUDGET;
    }
    cudaSetDevice(eng->device);
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        std::lock_guard<std::mutex> lk(eng->mu);
        if (give_back(eng)) {
            cudaGetLastError();
            e = cudaMalloc(p, bytes);
        }
    }
    if (e == cudaSuccess)
        return CMD_OK;
    budget_give(eng, bytes);
    return cuda_fail(e, what);
}

int Scratch::reserve(cmd_engine *eng, size_t bytes, int no_memory)
{
    if (bytes <= cap)
        return CMD_OK;
    BesideCapture beside;
    size_t want = align_up(std::max(bytes, cap + cap / 2), 1 << 20);
    const bool staged = this == &eng->staged;
    const size_t held = captured ? 0 : cap;  // bytes charged that the new block replaces
    if (!budget_take(eng, want - held) && (staged || !give_back(eng) || !budget_take(eng, want - held))) {
        set_last_error("scratch growth exceeds the engine HBM budget");
        return CMD_E_BUDGET;
    }
    if (captured) {
        eng->graph_blocks.push_back(ptr);
        eng->graph_block_bytes += cap;
        captured = false;
    } else if (ptr) {
        if (done)
            cudaEventSynchronize(done);
        cudaFree(ptr);
    }
    ptr = nullptr;
    cudaError_t e = cudaMalloc(&ptr, want);
    if (e == cudaErrorMemoryAllocation && !staged && give_back(eng)) {
        cudaGetLastError();
        e = cudaMalloc(&ptr, want);
    }
    if (e != cudaSuccess) {
        budget_give(eng, want);
        ptr = nullptr;
        cap = 0;
        const int rc = cuda_fail(e, "cudaMalloc(scratch)");
        if (e != cudaErrorMemoryAllocation || no_memory == rc)
            return rc;
        cudaGetLastError();
        return no_memory;
    }
    cap = want;
    return CMD_OK;
}

bool capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess)
        return cap != cudaStreamCaptureStatusNone;
    cudaGetLastError();  // the legacy stream beside a capture
    return true;
}

int graph_alloc(cmd_engine *eng, size_t bytes, void **p)
{
    if (!budget_take(eng, bytes)) {
        set_last_error("graph's work lists exceed the engine HBM budget");
        return CMD_E_BUDGET;
    }
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        budget_give(eng, bytes);
        return cuda_fail(e, "cudaMalloc(graph)");
    }
    eng->graph_blocks.push_back(*p);
    eng->graph_block_bytes += bytes;
    return CMD_OK;
}

int Scratch::begin(cmd_engine *eng, size_t bytes, cudaStream_t s, int no_memory)
{
    const int rc = reserve(eng, bytes, no_memory);
    if (rc)
        return rc;
    if (capturing(s)) {
        captured = ptr != nullptr;
        return CMD_OK;
    }
    if (!done)
        return CMD_OK;
    const cudaError_t e = cudaStreamWaitEvent(s, done);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "scratch order");
}

int Scratch::end(cudaStream_t s, cudaError_t e)
{
    if (!capturing(s)) {
        cudaError_t r = done ? cudaSuccess : cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
        if (r == cudaSuccess)
            r = cudaEventRecord(done, s);
        if (e == cudaSuccess)
            e = r;
    }
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "batch on the engine's scratch");
}

void Scratch::release(cmd_engine *eng)
{
    if (done) {
        cudaEventSynchronize(done);
        cudaEventDestroy(done);
    }
    if (ptr)
        cudaFree(ptr);
    budget_give(eng, cap);
    ptr = nullptr;
    done = nullptr;
    captured = false;
    cap = 0;
}

// Bump allocation inside one scratch reservation (256-byte aligned slices).
struct Carver {
    uint8_t *base;
    size_t off = 0;
    template <class T> T *take(size_t count)
    {
        off = align_up(off, 256);
        T *p = reinterpret_cast<T *>(base + off);
        off += count * sizeof(T);
        return p;
    }
};
static size_t carve_size(std::initializer_list<size_t> sizes)
{
    size_t off = 0;
    for (size_t s : sizes)
        off = align_up(off, 256) + s;
    return off + 256;
}

}  // namespace cmd

using namespace cmd;

extern "C" {

const char *cmd_last_error(void) { return g_last_error.c_str(); }

int cmd_set_info_get(cmd_set set, cmd_set_info *out)
{
    if (!out || !valid_set(set))
        return CMD_E_ARG;
    SetInfo s = set_info(set);
    out->set_id = s.id;
    out->m = s.m;
    out->n = s.n;
    out->t = s.t;
    out->ct_bytes = s.ct;
    out->sk_bytes = s.sk;
    out->sb = s.sb;
    out->err_bytes = s.n / 8;
    out->err_words = s.nw;
    return CMD_OK;
}

int cmd_set_from_name(const char *name, cmd_set *out)
{
    if (!name || !out)
        return CMD_E_ARG;
    const char *p = name;
    if (!strncmp(p, "mceliece", 8))
        p += 8;
    for (int s = 0; s < NSETS; s++) {
        char buf[16];
        snprintf(buf, sizeof buf, "%d", set_info(s).id);
        if (!strcmp(p, buf)) {
            *out = (cmd_set)s;
            return CMD_OK;
        }
    }
    set_last_error(std::string("unknown parameter set: ") + name);
    return CMD_E_ARG;
}

int cmd_engine_create(int device, size_t hbm_budget_bytes, cmd_engine **out)
{
    if (!out)
        return CMD_E_ARG;
    *out = nullptr;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        set_last_error(e != cudaSuccess ? cudaGetErrorString(e) : "no CUDA device");
        return CMD_E_NODEVICE;
    }
    if (device < 0 || device >= ndev)
        return CMD_E_ARG;
    if ((e = cudaSetDevice(device)) != cudaSuccess)
        return cuda_fail(e, "cudaSetDevice");
    cudaDeviceProp prop;
    if ((e = cudaGetDeviceProperties(&prop, device)) != cudaSuccess)
        return cuda_fail(e, "cudaGetDeviceProperties");
    if (prop.major != 10) {
        set_last_error("this build targets sm_100a (B200); device is sm_" + std::to_string(prop.major) +
                       std::to_string(prop.minor));
        return CMD_E_NODEVICE;
    }
    cmd_engine *eng = new (std::nothrow) cmd_engine();
    if (!eng)
        return CMD_E_NOMEM;
    eng->device = device;
    eng->num_sms = prop.multiProcessorCount;
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    eng->budget = hbm_budget_bytes ? hbm_budget_bytes : free_b / 10 * 8;
    if ((e = cudaStreamCreateWithFlags(&eng->stream, cudaStreamNonBlocking)) != cudaSuccess) {
        delete eng;
        return cuda_fail(e, "cudaStreamCreate");
    }
    snprintf(eng->gpu_name, sizeof eng->gpu_name, "%s", prop.name);
    // now, since a launch may be captured, when nothing can be allocated
    if ((e = cudaMalloc(&eng->tile_counter, TILE_COUNTERS * 4)) != cudaSuccess) {
        cudaStreamDestroy(eng->stream);
        delete eng;
        return cuda_fail(e, "cudaMalloc(counters)");
    }
    if (int rc = noalloc_setup(device)) {
        cudaFree(eng->tile_counter);
        cudaStreamDestroy(eng->stream);
        delete eng;
        return rc;
    }
    if (int rc = upload_fft_plans(eng)) {
        cudaFree(eng->tile_counter);
        cudaStreamDestroy(eng->stream);
        delete eng;
        return rc;
    }
    *out = eng;
    return CMD_OK;
}

void cmd_engine_destroy(cmd_engine *eng)
{
    if (!eng)
        return;
    cudaSetDevice(eng->device);
    cudaStreamSynchronize(eng->stream);
    eng->scratch.release(eng);
    eng->io.release(eng);
    eng->fused.release(eng);
    eng->staged.release(eng);
    eng->keygen.release(eng);
    for (void *p : eng->graph_blocks)
        cudaFree(p);
    budget_give(eng, eng->graph_block_bytes);
    eng->host_scratch.release();
    release_fft_plans(eng);
    for (int i = 0; i < BATCH_STREAMS; i++)
        if (eng->piece_stream[i]) {
            cudaStreamSynchronize(eng->piece_stream[i]);
            cudaStreamDestroy(eng->piece_stream[i]);
        }
    if (eng->staged_fork)
        cudaEventDestroy(eng->staged_fork);
    for (cudaEvent_t ev : eng->staged_join)
        if (ev)
            cudaEventDestroy(ev);
    cudaFree(eng->tile_counter);
    for (cudaEvent_t ev : eng->counter_done)
        if (ev)
            cudaEventDestroy(ev);
    for (uint32_t *block : eng->graph_counters)
        cudaFree(block);
    cudaStreamDestroy(eng->stream);
    delete eng;
}

int cmd_engine_memory(const cmd_engine *eng, size_t *used, size_t *budget)
{
    if (!eng)
        return CMD_E_ARG;
    if (used)
        *used = eng->used.load();
    if (budget)
        *budget = eng->budget;
    return CMD_OK;
}

uint64_t cmd_engine_launch_count(const cmd_engine *eng) { return eng ? eng->launches.load() : 0; }

// ---------------------------------------------------------------- keys

int cmd_key_expand(cmd_engine *eng, cmd_set set, const uint8_t *h_sk, size_t sk_len, cmd_key **out)
{
    if (!eng || !h_sk || !out || !valid_set(set))
        return CMD_E_ARG;
    *out = nullptr;
    const SetInfo si = set_info(set);
    if (sk_len != (size_t)si.sk) {
        set_last_error("secret key must be exactly " + std::to_string(si.sk) + " bytes for set " +
                       std::to_string(si.id));
        return CMD_E_ARG;
    }
    const size_t bytes = carve_size({(size_t)si.n * 2, (size_t)(si.t + 1) * 2, (size_t)si.n * 2,
                                     (size_t)si.sb * si.twp() * 4, (size_t)si.sb * si.twd() * 4,
                                     (size_t)si.m * si.nw * 4,
                                     benes_mask_words(si) * 4, fft_weight_words(si) * 4, (size_t)si.sk});
    cmd_key *key = new (std::nothrow) cmd_key();
    if (!key)
        return CMD_E_NOMEM;
    key->eng = eng;
    key->bytes = bytes;
    if (const int rc = device_alloc(eng, &key->block, bytes, "cudaMalloc(key)", "key does not fit the engine HBM budget")) {
        delete key;
        return rc;
    }
    Carver cv{static_cast<uint8_t *>(key->block)};
    key->dev.set = set;
    key->dev.L = cv.take<uint16_t>(si.n);
    key->dev.g = cv.take<uint16_t>(si.t + 1);
    key->dev.ginv2 = cv.take<uint16_t>(si.n);
    key->dev.tab = cv.take<uint32_t>((size_t)si.sb * si.twp());
    key->dev.tabd = cv.take<uint32_t>((size_t)si.sb * si.twd());
    key->dev.Lbs = cv.take<uint32_t>((size_t)si.m * si.nw);
    key->dev.bctl = cv.take<uint32_t>(benes_mask_words(si));
    key->dev.wfft = cv.take<uint32_t>(fft_weight_words(si));
    key->dev.sk = cv.take<uint8_t>(si.sk);
    std::lock_guard<std::mutex> lk(eng->mu);
    cudaError_t e;
    if ((e = cudaMemcpyAsync(key->dev.sk, h_sk, si.sk, cudaMemcpyHostToDevice, eng->stream)) != cudaSuccess ||
        (e = launch_key_expand(key->dev, eng->stream, LaunchCounter{&eng->launches})) != cudaSuccess ||
        (e = cudaStreamSynchronize(eng->stream)) != cudaSuccess) {
        cudaFree(key->block);
        budget_give(eng, bytes);
        delete key;
        return cuda_fail(e, "key expansion");
    }
    *out = key;
    return CMD_OK;
}

void cmd_key_free(cmd_key *key)
{
    if (!key)
        return;
    cudaSetDevice(key->eng->device);
    cudaStreamSynchronize(key->eng->stream);
    cudaFree(key->block);
    budget_give(key->eng, key->bytes);
    if (key->pk) {
        cudaFree(key->pk);
        budget_give(key->eng, key->pk_bytes);
    }
    delete key;
}

int cmd_key_set(const cmd_key *key, cmd_set *out)
{
    if (!key || !out)
        return CMD_E_ARG;
    *out = (cmd_set)key->dev.set;
    return CMD_OK;
}

size_t cmd_key_device_bytes(const cmd_key *key) { return key ? key->bytes : 0; }

static int key_copy(const cmd_key *key, void *dst, const void *src, size_t bytes)
{
    cudaSetDevice(key->eng->device);
    cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "cudaMemcpy(key D2H)");
}

int cmd_key_support(const cmd_key *key, uint16_t *h_L, size_t n)
{
    if (!key || !h_L || n != (size_t)set_info(key->dev.set).n)
        return CMD_E_ARG;
    return key_copy(key, h_L, key->dev.L, n * 2);
}

int cmd_key_goppa(const cmd_key *key, uint16_t *h_g, size_t t_plus_1)
{
    if (!key || !h_g || t_plus_1 != (size_t)set_info(key->dev.set).t + 1)
        return CMD_E_ARG;
    return key_copy(key, h_g, key->dev.g, t_plus_1 * 2);
}

int cmd_key_synd_table(const cmd_key *key, uint16_t *h_tab, size_t entries)
{
    const SetInfo si = key ? set_info(key->dev.set) : SetInfo{};
    if (!key || !h_tab || entries != (size_t)si.sb * 2 * si.t)
        return CMD_E_ARG;
    cudaSetDevice(key->eng->device);
    cudaError_t e = cudaMemcpy2D(h_tab, (size_t)si.t * 4, key->dev.tab, (size_t)si.twp() * 4, (size_t)si.t * 4,
                                 si.sb, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "cudaMemcpy2D(table D2H)");
}

// ---------------------------------------------------------------- stages

int cmd_stage_synd(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint16_t *d_synd,
                   void *stream)
{
    if (!eng || !key || (count && (!d_cts || !d_synd)))
        return CMD_E_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : eng->stream;
    cudaError_t e = launch_synd_plain(key->dev, d_cts, count, reinterpret_cast<uint32_t *>(d_synd), s,
                                      LaunchCounter{&eng->launches});
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "synd kernel");
}

int cmd_stage_synd_fft(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint16_t *d_synd,
                       void *stream)
{
    if (!eng || !key || key->eng != eng || (count && (!d_cts || !d_synd)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    cudaSetDevice(eng->device);
    std::lock_guard<std::mutex> lk(eng->mu);
    return run_tile(eng, key, d_cts, count, nullptr, nullptr, nullptr, d_synd,
                    stream ? (cudaStream_t)stream : eng->stream, eng->scratch);
}

int cmd_stage_bm(cmd_engine *eng, cmd_set set, const uint16_t *d_synd, size_t count, uint16_t *d_loc, void *stream)
{
    if (!eng || !valid_set(set) || (count && (!d_synd || !d_loc)))
        return CMD_E_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : eng->stream;
    cudaError_t e = launch_bm_plain(set, d_synd, count, d_loc, s, LaunchCounter{&eng->launches});
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "bm kernel");
}

int cmd_stage_root(cmd_engine *eng, const cmd_key *key, const uint16_t *d_loc, size_t count, uint32_t *d_err,
                   uint16_t *d_weight, void *stream)
{
    if (!eng || !key || (count && (!d_loc || !d_err)))
        return CMD_E_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : eng->stream;
    cudaError_t e = launch_root_plain(key->dev, d_loc, count, d_err, d_weight, s, LaunchCounter{&eng->launches},
                                      eng->num_sms);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "root kernel");
}

int cmd_stage_root_images(cmd_engine *eng, const cmd_key *key, const uint16_t *d_loc, size_t count,
                          uint16_t *d_images, void *stream)
{
    if (!eng || !key || (count && (!d_loc || !d_images)))
        return CMD_E_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : eng->stream;
    cudaError_t e = launch_root_images(key->dev, d_loc, count, d_images, s, LaunchCounter{&eng->launches});
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "root images kernel");
}

// ---------------------------------------------------------------- batches

}  // extern "C"

namespace cmd {

// Scratch the plain path needs for a batch: per chunk of up to 2^18
// ciphertexts, the syndromes (t words) and locators (t+1 u16) of each.
size_t plain_scratch_bytes(int set, size_t count)
{
    const SetInfo si = set_info(set);
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 18);
    return carve_size({chunk * si.t * 4, chunk * (si.t + 1) * 2});
}

// Plain path over a device batch, in chunks so the syndrome/locator
// intermediates stay bounded.  Caller holds eng->mu.
static int run_plain(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                     uint16_t *d_weight, cudaStream_t s)
{
    const SetInfo si = set_info(key->dev.set);
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 18);
    const size_t need = plain_scratch_bytes(key->dev.set, count);
    int rc = eng->scratch.begin(eng, need, s);
    if (rc)
        return rc;
    Carver cv{static_cast<uint8_t *>(eng->scratch.ptr)};
    uint32_t *synd = cv.take<uint32_t>(chunk * si.t);
    uint16_t *loc = cv.take<uint16_t>(chunk * (si.t + 1));
    LaunchCounter lc{&eng->launches};
    cudaError_t e = cudaSuccess;
    for (size_t c0 = 0; c0 < count && e == cudaSuccess; c0 += chunk) {
        const size_t n = std::min(chunk, count - c0);
        if ((e = launch_synd_plain(key->dev, d_cts + c0 * si.ct, n, synd, s, lc)) != cudaSuccess ||
            (e = launch_bm_plain(key->dev.set, reinterpret_cast<uint16_t *>(synd), n, loc, s, lc)) != cudaSuccess ||
            (e = launch_root_plain(key->dev, loc, n, d_err + c0 * si.nw, d_weight ? d_weight + c0 : nullptr, s, lc,
                                   eng->num_sms)) != cudaSuccess)
            break;
    }
    return eng->scratch.end(s, e);
}

// The serving tile kernels over one key's batch, in chunks whose byte and
// word offsets fit the tile items' 32-bit fields.  With d_synd: syndromes
// only.  buf: the engine's scratch, or that of the staged batches.  Caller holds
// eng->mu.
static int run_tile(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                    uint16_t *d_weight, uint16_t *d_pos, uint16_t *d_synd, cudaStream_t s, Scratch &buf)
{
    const SetInfo si = set_info(key->dev.set);
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 22);
    const bool on_chip = !d_synd && count <= CT_ONE_LAUNCH;  // one launch, no scratch
    if (!on_chip)
        if (const int rc = buf.begin(eng, tile_single_scratch_words(chunk) * 4, s,
                                     &buf == &eng->staged ? CMD_E_BUDGET : CMD_E_CUDA))
            return rc;
    uint32_t *scratch = on_chip ? nullptr : static_cast<uint32_t *>(buf.ptr);
    FftPlans plans;
    for (int st = 0; st < NSETS; st++)
        plans.p[st] = eng->fft[st];
    cudaError_t e = cudaSuccess;
    for (size_t c0 = 0; c0 < count && e == cudaSuccess; c0 += chunk) {
        const size_t n = std::min(chunk, count - c0);
        e = launch_tile_single(
            key->dev, d_cts + c0 * si.ct, n, scratch, d_err ? d_err + c0 * si.nw : nullptr,
            d_weight ? d_weight + c0 : nullptr, d_pos,
            d_synd ? d_synd + c0 * 2 * si.t : nullptr, plans, eng->num_sms, s, LaunchCounter{&eng->launches});
    }
    if (!on_chip)
        return buf.end(s, e);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "tile path launch");
}

int ensure_piece_streams(cmd_engine *eng)
{
    for (int i = 0; i < BATCH_STREAMS; i++)
        if (!eng->piece_stream[i]) {
            const cudaError_t e = cudaStreamCreateWithFlags(&eng->piece_stream[i], cudaStreamNonBlocking);
            if (e != cudaSuccess)
                return cuda_fail(e, "cudaStreamCreate(piece)");
        }
    return CMD_OK;
}

// Parts of a staged batch (sizes for 148 SMs, the only part this library is built
// for; measured with mceliece6960119): one up to 45,000 ciphertexts (about a wave of
// Berlekamp-Massey warps), two equal ones up to 131,072, then parts of about
// 65,536.  Parts run on their own streams, STAGED_STREAMS in flight, so that one
// part's syndromes (shared-memory bound) and ends of waves run beside another's
// Berlekamp-Massey and FFT (logic bound): 65,536 mceliece6960119 ciphertexts
// 2,709 us in one part, 2,537 us in two; 262,144 10,527 us in one stream's
// parts of 131,072, 9,642 us in four of 65,536.
static size_t staged_part(size_t count)
{
    const size_t parts = count <= 45000 ? 1 : count <= 131072 ? 2 : (count + 65535) / 65536;
    return ((count + parts - 1) / parts + 31) / 32 * 32;
}

int staged_begin(cmd_engine *eng, size_t bytes, int ns, cudaStream_t s)
{
    int rc = eng->staged.begin(eng, bytes, s, CMD_E_BUDGET);
    if (rc || ns == 1)
        return rc;
    if ((rc = ensure_piece_streams(eng)))
        return rc;
    cudaError_t e = cudaSuccess;
    auto make = [&](cudaEvent_t &ev) {
        if (!ev && e == cudaSuccess)
            e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    };
    make(eng->staged_fork);
    for (cudaEvent_t &ev : eng->staged_join)
        make(ev);
    if (e == cudaSuccess)
        e = cudaEventRecord(eng->staged_fork, s);
    for (int i = 0; i < ns && e == cudaSuccess; i++)
        e = cudaStreamWaitEvent(eng->piece_stream[i], eng->staged_fork);
    return e == cudaSuccess ? CMD_OK : cuda_fail(e, "staged batch");
}

int staged_end(cmd_engine *eng, int ns, cudaStream_t s, cudaError_t e)
{
    for (int i = 0; i < ns && ns > 1; i++) {  // joined even after an error
        cudaError_t e2 = cudaEventRecord(eng->staged_join[i], eng->piece_stream[i]);
        if (e2 == cudaSuccess)
            e2 = cudaStreamWaitEvent(s, eng->staged_join[i]);
        if (e == cudaSuccess)
            e = e2;
    }
    return eng->staged.end(s, e);
}

int run_staged(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
               uint16_t *d_weight, uint16_t *d_pos, cudaStream_t s)
{
    const SetInfo si = set_info(key->dev.set);
    const size_t part = staged_part(count), nparts = (count + part - 1) / part;
    const size_t ns = std::min<size_t>(nparts, STAGED_STREAMS), words = staged_scratch_words(key->dev.set, part);
    if (const int rc = staged_begin(eng, ns * words * 4, (int)ns, s))
        return rc;
    cudaError_t e = cudaSuccess;
    for (size_t p = 0; p < nparts && e == cudaSuccess; p++) {
        const size_t c0 = p * part, n = std::min(part, count - c0), i = p % ns;
        e = launch_staged(key->dev, d_cts + c0 * si.ct, (uint32_t)n,
                          static_cast<uint32_t *>(eng->staged.ptr) + i * words, d_err ? d_err + c0 * si.nw : nullptr,
                          d_weight ? d_weight + c0 : nullptr, d_pos ? d_pos + c0 * (si.t + 1) : nullptr,
                          eng->fft[key->dev.set], eng->num_sms, nparts > 2, ns > 1 ? eng->piece_stream[i] : s,
                          LaunchCounter{&eng->launches});
    }
    return staged_end(eng, (int)ns, s, e);
}

// Whether CMD_PATH_AUTO takes the small-batch kernels: batches within the
// per-ciphertext kernels' reach, or below the tuned crossover.  At 24 ciphertexts
// an SM (3,552) the per-ciphertext kernels and the staged ones take the same time
// (6960119 438 and 447 us, 348864 205 and 235 us), at half of that 279 against
// 415 us; the fused kernel takes 1,037 us for any number up to 18,944.
static bool takes_small(const cmd_engine *eng, int set, size_t count)
{
    return count <= (size_t)CT_PER_SM * eng->num_sms || count < eng->fcfg[set].tile_below;
}

// The best kernels for the batch size, error rows and weights or positions:
// small-batch kernels, else the staged ones.  The fused kernel takes batches of
// six to eight tiles an SM, one nearly full round of its warps (37,888
// mceliece6960119 ciphertexts 1,485 us, staged 1,534 us); needing no scratch, it
// also runs when theirs does not fit the budget or the device's free memory, and
// under stream capture, where nothing may be allocated and a graph would keep the
// address of scratch that can grow.
static int run_auto(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                    uint16_t *d_weight, uint16_t *d_pos, cudaStream_t s)
{
    const int set = key->dev.set;
    if (!capturing(s)) {
        if (takes_small(eng, set, count) && (!d_pos || count <= (size_t)CT_PER_SM * eng->num_sms)) {
            const int rc = run_tile(eng, key, d_cts, count, d_err, d_weight, d_pos, nullptr, s, eng->staged);
            if (rc != CMD_E_BUDGET)
                return rc;
        } else if (count <= 192 * (size_t)eng->num_sms || count > 256 * (size_t)eng->num_sms) {
            const int rc = run_staged(eng, key, d_cts, count, d_err, d_weight, d_pos, s);
            if (rc != CMD_E_BUDGET)
                return rc;
        }
    }
    cudaGetLastError();
    return run_fused_single(eng, key, d_cts, count, d_err, d_weight, s, d_pos);
}

int run_device(cmd_engine *eng, const cmd_key *key, cmd_path path, const uint8_t *d_cts, size_t count,
               uint32_t *d_err, uint16_t *d_weight, cudaStream_t s, uint16_t *d_pos)
{
    if (count == 0)
        return CMD_OK;
    if (path == CMD_PATH_PLAIN)
        return run_plain(eng, key, d_cts, count, d_err, d_weight, s);
    if (path == CMD_PATH_TILE)
        return run_tile(eng, key, d_cts, count, d_err, d_weight, nullptr, nullptr, s, eng->scratch);
    if (path == CMD_PATH_AUTO)
        return run_auto(eng, key, d_cts, count, d_err, d_weight, d_pos, s);
    return run_fused_single(eng, key, d_cts, count, d_err, d_weight, s);
}

// A device address through which kernels can write the host range [h, h +
// bytes), or null: pinned memory the GPU maps (cudaHostAlloc / cudaMallocHost
// memory under unified addressing, or registered memory with a device
// mapping), 2-byte aligned, whose first and last bytes map to one contiguous
// device range.  Anything else (pageable memory, a range running past its
// pinned allocation) gives null, and the caller copies through staging.
uint8_t *device_view(uint8_t *h, size_t bytes)
{
    if (!h || !bytes || (((uintptr_t)h) & 1))
        return nullptr;
    cudaPointerAttributes a0{}, a1{};
    if (cudaPointerGetAttributes(&a0, h) != cudaSuccess || a0.type != cudaMemoryTypeHost || !a0.devicePointer) {
        cudaGetLastError();
        return nullptr;
    }
    if (cudaPointerGetAttributes(&a1, h + bytes - 1) != cudaSuccess || a1.type != cudaMemoryTypeHost ||
        static_cast<uint8_t *>(a1.devicePointer) != static_cast<uint8_t *>(a0.devicePointer) + (bytes - 1)) {
        cudaGetLastError();
        return nullptr;
    }
    return static_cast<uint8_t *>(a0.devicePointer);
}

}  // namespace cmd

extern "C" {

int cmd_decrypt_device(cmd_engine *eng, const cmd_key *key, cmd_path path, const uint8_t *d_cts, size_t count,
                       uint32_t *d_err, uint16_t *d_weight, void *stream)
{
    if (!eng || !key || key->eng != eng || (count && (!d_cts || !d_err)) || path < 0 || path > 3)
        return CMD_E_ARG;
    cudaSetDevice(eng->device);
    std::lock_guard<std::mutex> lk(eng->mu);
    return run_device(eng, key, path, d_cts, count, d_err, d_weight, stream ? (cudaStream_t)stream : eng->stream);
}


int cmd_decrypt_batch(cmd_engine *eng, const cmd_key *key, cmd_path path, const uint8_t *h_cts, size_t count,
                      uint8_t *h_err, uint16_t *h_weight)
{
    if (!eng || !key || key->eng != eng || (count && (!h_cts || !h_err)) || path < 0 || path > 3)
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    cudaSetDevice(eng->device);
    const SetInfo si = set_info(key->dev.set);
    std::lock_guard<std::mutex> lk(eng->mu);
    // Device staging: ciphertexts, error rows, weights; processed in chunks so
    // the staging stays bounded for very large host batches.
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 20);
    const size_t need = carve_size({chunk * si.ct, chunk * si.nw * 4, chunk * 2});
    int rc = eng->io.reserve(eng, need);
    if (rc)
        return rc;
    Carver cv{static_cast<uint8_t *>(eng->io.ptr)};
    uint8_t *d_cts = cv.take<uint8_t>(chunk * si.ct);
    uint32_t *d_err = cv.take<uint32_t>(chunk * si.nw);
    uint16_t *d_w = cv.take<uint16_t>(chunk);
    cudaStream_t s = eng->stream;
    // Large batches go as BATCH_STREAMS fused pieces on their own streams (each
    // with its own work counter, full rounds): one piece's copies run while the
    // others compute, and the pieces' kernels share the SMs.  The fused kernel
    // rather than the staged ones, because its rows come out evenly over its run:
    // staged pieces that fill the GPU end together, and their copies out follow
    // (100,003 mceliece6960119 ciphertexts 5.2 to 6.2 ms against 4.9 ms).
    const bool pieces = path != CMD_PATH_PLAIN && path != CMD_PATH_TILE && chunk >= (size_t)BATCH_STREAMS * 8192;
    // With host error rows the GPU can write, the pieces' kernels store the
    // packed rows there directly: the rows cross PCIe while the kernels run,
    // instead of in a copy after the last piece's kernel.
    uint8_t *err_view = pieces ? device_view(h_err, count * (size_t)(si.n / 8)) : nullptr;
    if (pieces && (rc = ensure_piece_streams(eng)))
        return rc;
    for (size_t c0 = 0; c0 < count; c0 += chunk) {
        const size_t n = std::min(chunk, count - c0);
        if (pieces) {
            // pieces of whole rounds of the size one launch over the chunk
            // would use (equal shares per resident CTA when so tuned), so the
            // pieces' rounds fill the same waves; a round is a multiple of 32
            // ciphertexts, so every piece's ciphertexts start 16-byte aligned
            const uint32_t round = fused_round(eng, key->dev.set, n);
            const size_t per = (n + (size_t)BATCH_STREAMS * round - 1) / ((size_t)BATCH_STREAMS * round) * round;
            cudaError_t e = cudaSuccess;
            for (int i = 0; i < BATCH_STREAMS && e == cudaSuccess && rc == CMD_OK; i++) {
                const size_t p0 = (size_t)i * per;
                if (p0 >= n)
                    break;
                const size_t pn = std::min(per, n - p0);
                cudaStream_t ps = eng->piece_stream[i];
                e = cudaMemcpyAsync(d_cts + p0 * si.ct, h_cts + (c0 + p0) * si.ct, pn * si.ct, cudaMemcpyHostToDevice,
                                    ps);
                if (e != cudaSuccess)
                    break;
                uint8_t *pack = err_view ? err_view + (c0 + p0) * (size_t)(si.n / 8) : nullptr;
                rc = run_fused_counter(eng, key, d_cts + p0 * si.ct, pn, pack ? nullptr : d_err + p0 * si.nw,
                                       d_w + p0, ps, eng->tile_counter + 1 + i, nullptr, 0, round, pack);
                if (rc)
                    break;
                if (!pack)
                    e = cudaMemcpy2DAsync(h_err + (c0 + p0) * (si.n / 8), si.n / 8, d_err + p0 * si.nw,
                                          (size_t)si.nw * 4, si.n / 8, pn, cudaMemcpyDeviceToHost, ps);
                if (e == cudaSuccess && h_weight)
                    e = cudaMemcpyAsync(h_weight + c0 + p0, d_w + p0, pn * 2, cudaMemcpyDeviceToHost, ps);
            }
            for (int i = 0; i < BATCH_STREAMS; i++) {
                const cudaError_t e2 = cudaStreamSynchronize(eng->piece_stream[i]);
                if (e == cudaSuccess)
                    e = e2;
            }
            if (rc)
                return rc;
            if (e != cudaSuccess)
                return cuda_fail(e, "decrypt batch pieces");
            continue;
        }
        cudaError_t e = cudaMemcpyAsync(d_cts, h_cts + c0 * si.ct, n * si.ct, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMemcpyAsync(cts H2D)");
        if ((rc = run_device(eng, key, path, d_cts, n, d_err, d_w, s)))
            return rc;
        // Strip the word padding of each row: n/8 bytes per vector on the host.
        e = cudaMemcpy2DAsync(h_err + c0 * (si.n / 8), si.n / 8, d_err, (size_t)si.nw * 4, si.n / 8, n,
                              cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && h_weight)
            e = cudaMemcpyAsync(h_weight + c0, d_w, n * 2, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(s);
        if (e != cudaSuccess)
            return cuda_fail(e, "decrypt batch D2H");
    }
    return CMD_OK;
}

int cmd_decrypt_positions_device(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count,
                                 uint16_t *d_pos, void *stream)
{
    if (!eng || !key || key->eng != eng || (count && (!d_cts || !d_pos)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    cudaSetDevice(eng->device);
    std::lock_guard<std::mutex> lk(eng->mu);
    return run_device(eng, key, CMD_PATH_AUTO, d_cts, count, nullptr, nullptr,
                      stream ? (cudaStream_t)stream : eng->stream, d_pos);
}

int cmd_decrypt_positions(cmd_engine *eng, const cmd_key *key, const uint8_t *h_cts, size_t count, uint16_t *h_pos)
{
    if (!eng || !key || key->eng != eng || (count && (!h_cts || !h_pos)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    cudaSetDevice(eng->device);
    const SetInfo si = set_info(key->dev.set);
    const size_t row = (size_t)si.t + 1;
    std::lock_guard<std::mutex> lk(eng->mu);
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 20);
    const size_t need = carve_size({chunk * si.ct, chunk * row * 2});
    int rc = eng->io.reserve(eng, need);
    if (rc)
        return rc;
    Carver cv{static_cast<uint8_t *>(eng->io.ptr)};
    uint8_t *d_cts = cv.take<uint8_t>(chunk * si.ct);
    uint16_t *d_pos = cv.take<uint16_t>(chunk * row);
    cudaStream_t s = eng->stream;
    const bool pieces = chunk >= (size_t)BATCH_STREAMS * 8192;
    if (pieces && (rc = ensure_piece_streams(eng)))
        return rc;
    for (size_t c0 = 0; c0 < count; c0 += chunk) {
        const size_t n = std::min(chunk, count - c0);
        if (pieces) {  // as in cmd_decrypt_batch
            const uint32_t round = fused_round(eng, key->dev.set, n);
            const size_t per = (n + (size_t)BATCH_STREAMS * round - 1) / ((size_t)BATCH_STREAMS * round) * round;
            cudaError_t e = cudaSuccess;
            for (int i = 0; i < BATCH_STREAMS && e == cudaSuccess && rc == CMD_OK; i++) {
                const size_t p0 = (size_t)i * per;
                if (p0 >= n)
                    break;
                const size_t pn = std::min(per, n - p0);
                cudaStream_t ps = eng->piece_stream[i];
                e = cudaMemcpyAsync(d_cts + p0 * si.ct, h_cts + (c0 + p0) * si.ct, pn * si.ct, cudaMemcpyHostToDevice,
                                    ps);
                if (e != cudaSuccess)
                    break;
                rc = run_fused_counter(eng, key, d_cts + p0 * si.ct, pn, nullptr, nullptr, ps,
                                       eng->tile_counter + 1 + i, d_pos + p0 * row, 0, round);
                if (rc)
                    break;
                e = cudaMemcpyAsync(h_pos + (c0 + p0) * row, d_pos + p0 * row, pn * row * 2, cudaMemcpyDeviceToHost,
                                    ps);
            }
            for (int i = 0; i < BATCH_STREAMS; i++) {
                const cudaError_t e2 = cudaStreamSynchronize(eng->piece_stream[i]);
                if (e == cudaSuccess)
                    e = e2;
            }
            if (rc)
                return rc;
            if (e != cudaSuccess)
                return cuda_fail(e, "decrypt positions pieces");
            continue;
        }
        cudaError_t e = cudaMemcpyAsync(d_cts, h_cts + c0 * si.ct, n * si.ct, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMemcpyAsync(cts H2D)");
        if ((rc = run_device(eng, key, CMD_PATH_AUTO, d_cts, n, nullptr, nullptr, s, d_pos)))
            return rc;
        e = cudaMemcpyAsync(h_pos + c0 * row, d_pos, n * row * 2, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(s);
        if (e != cudaSuccess)
            return cuda_fail(e, "decrypt positions D2H");
    }
    return CMD_OK;
}

}  // extern "C"

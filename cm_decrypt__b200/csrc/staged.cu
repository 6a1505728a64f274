// Staged decrypt of one key's batch, or of a mixed batch set by set (MIX below:
// the slots of a tile belong to one key): the fused kernel's phases as four kernels,
// each with the block shape, shared memory and code size that its phase wants.
//
//   k_synd_table  the 2t syndromes (util.c:102-114) from the key's dense table,
//                 lane = ciphertext, rows five at a time;
//   k_bm_tile     Berlekamp-Massey (bm.c:12-68), a warp and block per tile of 32
//                 ciphertexts, and the locators' radix conversion (k_bm_pair: per
//                 two tiles);
//   k_fft_tile    the locators at all field elements (additive FFT), a warp per
//                 ciphertext: zero flags;
//   k_net_rows    the key's support network (root_13.c:95-177) over the flags of
//                 four ciphertexts at a time, and the outputs.
//
// The fused kernel keeps a tile's data on chip from end to end, but a CTA's
// eight warps then move through the phases together: the syndrome phase waits on
// shared memory with the logic pipe idle, the root search runs at the
// Berlekamp-Massey phase's eight warps an SM, the instruction caches hold the
// code of all phases, and a batch is cut into whole rounds of 256 ciphertexts an
// SM.  The intermediates that go through memory here are small: 416 bytes a
// ciphertext (syndromes, then the converted locator) and 1 KB of flags.
//
// Measured on a B200 against the fused kernel: 65,536 mceliece6960119 ciphertexts
// 2,830 -> 2,522 us, 50,000 of 8192128 3,036 -> 2,558 us, 2^20 of 348864 14.68 ->
// 12.69 ms, 12,345 of 460896 879 -> 642 us, 4,736 of 6960119 1,037 -> 440 us.  Of
// 37,888 ciphertexts of 6960119 in one part: syndromes 244 us (shared-memory
// bound), Berlekamp-Massey 820 us (logic pipe 85 % busy), FFT 467 us (89 %),
// network 43 us.
#include <algorithm>

#include "bm_tile.cuh"
#include "fft_root.cuh"
#include "internal.h"

namespace cmd {

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr int SYND_WARPS = 16;  // most warps of a k_synd_table block
constexpr int FFT_WARPS = 4;    // warps of a k_fft_tile block (one tile)
constexpr int NET_WARPS = 8;    // warps of a k_net_rows block

template <int S> struct SgDims {
    using P = Set<S>;
    static constexpr int M = P::M, T = P::T, SS = BmDims<S>::SS, TWD = P::TWD;
    static constexpr int NX = FftDims<S>::NX, NWD = FftDims<S>::NWD;
    static constexpr int TILE_WORDS = BmDims<S>::SYN_WORDS > NX * SS ? BmDims<S>::SYN_WORDS : NX * SS;
    static constexpr int BM_WORDS = 2 * BmDims<S>::RING_WORDS + BmDims<S>::C_WORDS;  // shared, per tile
    static_assert(NX * SS <= BM_WORDS && 4 * (BM_WORDS + 128) <= 48 * 1024, "conversion array in the same memory");
    static constexpr int PAIR_WORDS = (BM_WORDS + 15) / 32 * 32 + 16;  // a tile of a pair: 16 mod 32 (bm_tile)
    // two pairs a scheduler fit the SM's shared memory
    static constexpr bool PAIRS = 8 * (8 * PAIR_WORDS + 1024) <= 228 * 1024;
    static_assert(!PAIRS || 8 * PAIR_WORDS <= 48 * 1024, "no opt-in for shared memory");
    static constexpr int NWU = (2 * T * M + 31) / 32;  // syndrome words of a ciphertext
    // syndrome kernel: rows per group, combination rows an odd stride apart
    static constexpr int G = 5, NG = (P::SB + G - 1) / G, CS = NWU | 1, COMBS = 1 << G;
    static constexpr int ROW_BUFS = 8;  // groups of rows in flight or in use
    static constexpr int ROW_WORDS = ROW_BUFS * G * TWD, COMB_WORDS = 2 * COMBS * CS;
    static_assert(G == 5 && NWU <= 128, "forming the combinations: two parts of 128 words");
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}

// Syndromes.  Lane q of a warp keeps the 2t*m syndrome bits of its ciphertext in
// NWU registers.  The table rows go five at a time: the block forms the 32 XOR
// combinations of a group and each lane adds the one its ciphertext's five
// (public) bits select.  Combination rows lie an odd number of words apart, so
// the 32 rows start in 32 banks and every such load is one wavefront whatever
// the lanes pick (with six rows a group, combinations x and x + 32 share banks:
// 337 us against 244 us for 37,888 mceliece6960119 ciphertexts).  Combinations are
// double-buffered, group g + 1's formed beside group g's additions, one barrier a
// group; rows come in six groups ahead.  Bound by the shared loads (97 + 5 words
// a warp and group for t = 119 with 16 warps a block).
//
// blockDim.x = 32 * SPLIT * (tiles per block): SPLIT warps share the syndrome
// words of a tile: 8 up to two tiles an SM, 4 up to four, where a warp's time per
// group counts (4,736 ciphertexts: 452 us with one warp a tile, 137 us with four).
template <int S, int SPLIT, bool MIX = false>
__global__ void __launch_bounds__(SYND_WARPS * 32, 1) k_synd_table(const uint32_t *__restrict__ tab,
                                                                   const uint8_t *__restrict__ cts, uint32_t count,
                                                                   uint32_t *__restrict__ tiles, StagedMixed mx)
{
    using Z = SgDims<S>;
    using P = Set<S>;
    constexpr int NWU = Z::NWU, G = Z::G, TWD = Z::TWD, CS = Z::CS, M = Z::M;
    constexpr int NP = (NWU + SPLIT - 1) / SPLIT;  // words of one part
    extern __shared__ __align__(16) uint32_t smem_sg[];
    uint32_t *rows = smem_sg, *comb = rows + Z::ROW_WORDS;
    uint8_t *raw = reinterpret_cast<uint8_t *>(comb + Z::COMB_WORDS);
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const int part = (tid >> 5) % SPLIT, mine = (tid >> 5) / SPLIT * 32 + lane;  // ciphertext in the block
    const int nct = nt / SPLIT;                                                  // ciphertexts of a block
    uint64_t first = (uint64_t)blockIdx.x * nct, tile0 = first / 32;
    int live = (int)(count - first < (uint64_t)nct ? count - first : nct);
    if constexpr (MIX) {
        const StagedPiece blk = mx.blocks[blockIdx.x];
        tab = mx.keys[blk.key].tab;
        first = blk.first;
        tile0 = blk.tile0;
        live = (int)blk.count;
    }

    constexpr int AHEAD = Z::ROW_BUFS - 2;  // group g's additions, g + 1's combinations, the rest in flight
    auto stage = [&](int g) {  // rows of group g, zero past the last one
        for (int v = tid; v < G * TWD / 4 && g < Z::NG; v += nt) {
            uint32_t *dst = rows + (g % Z::ROW_BUFS) * G * TWD + 4 * v;
            if (g * G + v / (TWD / 4) < P::SB)
                cp_async16(dst, tab + (size_t)g * G * TWD + 4 * v);
            else
                *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto form = [&](int g) {  // its 32 combinations: word v & 127, the 16 with the fifth row in or out
        const uint32_t *src = rows + (g % Z::ROW_BUFS) * G * TWD;
        uint32_t *dst = comb + (g & 1) * Z::COMBS * CS;
        for (int v = tid; v < 256; v += nt) {
            const int w = v & 127, part = v >> 7;
            if (w >= NWU)
                continue;
            uint32_t c[16];
            c[0] = part ? src[4 * TWD + w] : 0u;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const uint32_t x = src[r * TWD + w];
#pragma unroll
                for (int i = 0; i < 1 << r; i++)
                    c[(1 << r) + i] = c[i] ^ x;
            }
            uint32_t *o = dst + (16 * part) * CS + w;
#pragma unroll
            for (int i = 0; i < 16; i++)
                o[i * CS] = c[i];
        }
    };

    for (int g = 0; g < AHEAD; g++)
        stage(g);
    uint16_t *dst16 = reinterpret_cast<uint16_t *>(raw);
    if constexpr (MIX) {  // a ciphertext starts at any byte
        for (int q = tid >> 5; q < live; q += nt >> 5) {
            const uint8_t *src = cts + mx.ct_off[mx.order[first + q]];
            for (int v = lane; v < P::CT; v += 32)
                raw[q * P::CT + v] = __ldg(src + v);
        }
        for (int v = live * P::CT / 2 + tid; v < nct * P::CT / 2 + 4; v += nt)
            dst16[v] = 0;
    } else {  // the block's ciphertexts: 16-bit loads (every set's length is even)
        const uint16_t *src = reinterpret_cast<const uint16_t *>(cts + first * P::CT);
        uint16_t *dst = dst16;
        if (((uintptr_t)src & 15) == 0) {
            const int n = live * P::CT / 16;
            for (int v = tid; v < n; v += nt)
                reinterpret_cast<uint4 *>(raw)[v] = __ldg(reinterpret_cast<const uint4 *>(src) + v);
            for (int v = 8 * n + tid; v < live * P::CT / 2; v += nt)
                dst[v] = __ldg(src + v);
        } else if (((uintptr_t)src & 1) == 0) {
            for (int v = tid; v < live * P::CT / 2; v += nt)
                dst[v] = __ldg(src + v);
        } else {
            for (int v = tid; v < live * P::CT; v += nt)
                raw[v] = __ldg(cts + first * P::CT + v);
        }
        for (int v = live * P::CT / 2 + tid; v < nct * P::CT / 2 + 4; v += nt)
            dst[v] = 0;  // absent ciphertexts, and the tail that the bit reads may touch
    }
    asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD - 2) : "memory");  // groups 0 and 1
    __syncthreads();
    form(0);
    __syncthreads();

    uint32_t acc[NP];
#pragma unroll
    for (int w = 0; w < NP; w++)
        acc[w] = 0;
    const uint32_t my = (uint32_t)mine * P::CT;  // byte offset of this lane's ciphertext
    const uint32_t *raw32 = reinterpret_cast<const uint32_t *>(raw);
#pragma unroll 1
    for (int g = 0; g < Z::NG; g++) {
        stage(g + AHEAD);
        if (g + 1 < Z::NG)
            form(g + 1);
        const uint32_t bit = 8 * my + g * G;
        const uint32_t x = __funnelshift_r(raw32[bit >> 5], raw32[(bit >> 5) + 1], bit & 31) & (Z::COMBS - 1);
        const uint32_t *pick = comb + (g & 1) * Z::COMBS * CS + x * CS + part * NP;
#pragma unroll
        for (int w = 0; w < NP; w++)
            if (SPLIT == 1 || part * NP + w < NWU)
                acc[w] ^= pick[w];
        asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD - 2) : "memory");  // up to group g + 2
        __syncthreads();
    }
    // transpose to bitsliced syndromes (bit q = ciphertext q of the tile), as in
    // the fused kernel: word x = j*m + k goes to row j
    const int ltile = (tid >> 5) / SPLIT;
    const uint64_t tile = tile0 + ltile;
    if (32 * ltile >= live)
        return;
    uint32_t *out = tiles + tile * Z::TILE_WORDS;
    constexpr uint32_t M0[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int w = 0; w < NP; w++) {
        uint32_t v = acc[w];
#pragma unroll
        for (int st = 0; st < 5; st++) {
            const int j = 16 >> st;
            const uint32_t y = __shfl_xor_sync(FULL, v, j);
            const uint32_t keep = (lane & j) ? ~M0[st] : M0[st];
            const uint32_t t = (lane & j) ? (y >> j) : (y << j);
            v = (v & keep) | (t & ~keep);
        }
        const int x = 32 * (part * NP + w) + lane;
        if (x < 2 * Z::T * M)
            out[Z::SS == M ? x : x / M * Z::SS + x % M] = v;
    }
}

// Berlekamp-Massey of one tile by W warps (bm_tile.cuh), then the radix
// conversion; the converted locators replace the syndromes in the tile's rows.
// One tile a block: tiles go to SMs one by one as blocks finish, so a batch has
// no rounds.  Bound by the logic pipe with eight or more warps an SM, by a step's
// latency with fewer; 19 KB of shared memory a tile.
template <int S, int W>
__global__ void __launch_bounds__(32 * W) k_bm_tile(uint32_t *__restrict__ tiles, uint32_t count,
                                                    const uint16_t *__restrict__ scalpow, uint32_t turn_after,
                                                    const StagedPiece *__restrict__ pieces)
{
    using Z = SgDims<S>;
    using B = BmDims<S>;
    constexpr int T = Z::T, SS = Z::SS, NX = Z::NX, NT = 32 * W;
    extern __shared__ __align__(16) uint32_t smem_sg[];
    const int tid = threadIdx.x;
    uint32_t *share = smem_sg, *ring = share + 2 * W * 16, *cm = ring + B::RING_WORDS, *syn = cm + B::C_WORDS;
    uint32_t *cv = ring;  // conversion array: the ring, C and the syndromes are free by then
    uint32_t *io = tiles + (size_t)blockIdx.x * Z::TILE_WORDS;
    const uint32_t left = pieces ? pieces[blockIdx.x].count : count - 32 * blockIdx.x;
    bm_tile<S, true, W>(syn, ring, cm, left < 32 ? (int)left : 32, tid, io, share,
                        W == 1 ? 0 : blockIdx.x / turn_after % W);
    // entry x of the conversion array is C[T-x] (bm.c:62-65 reverses the
    // locator), zero for T < x < 2^D; through the tile's rows in memory, since
    // the array overlaps C
    for (int v = tid; v < (T + 1) * SS; v += NT) {
        const int i = v / SS, k = v - i * SS;
        io[(T - i) * SS + k] = cm[v];
    }
    __syncthreads();
    for (int v = tid; v < NX * SS; v += NT)
        cv[v] = v < (T + 1) * SS ? io[v] : 0u;
    __syncthreads();
    fft_convert<S, SS, NT>(cv, scalpow, tid, [] { __syncthreads(); });
    for (int v = tid; v < NX * SS; v += NT)
        io[v] = cv[v];
}

// The same for two tiles by one warp (bm_tile's PAIR), for large batches of a set
// with room for ten pairs an SM: 2^20 mceliece348864 ciphertexts 13,397 -> 12,687
// us, 200,000 2,557 -> 2,463 us.
template <int S>
__global__ void __launch_bounds__(32) k_bm_pair(uint32_t *__restrict__ tiles, uint32_t ntiles, uint32_t count,
                                                const uint16_t *__restrict__ scalpow)
{
    using Z = SgDims<S>;
    using B = BmDims<S>;
    constexpr int T = Z::T, SS = Z::SS, NX = Z::NX, HW = Z::PAIR_WORDS;
    extern __shared__ __align__(16) uint32_t smem_sg[];
    const int lane = threadIdx.x;
    const uint32_t tile0 = 2 * blockIdx.x;
    const int nt = ntiles - tile0 < 2 ? 1 : 2;  // for an absent second tile, the first's again, not stored
    const uint32_t tile = tile0 + (nt == 2 ? lane >> 4 : 0);
    uint32_t *ring = smem_sg + (lane >> 4) * HW, *cm = ring + B::RING_WORDS, *syn = cm + B::C_WORDS;
    const uint32_t left = count - 32 * tile;
    bm_tile<S, true, 1, true>(syn, ring, cm, left < 32 ? (int)left : 32, lane,
                              tiles + (size_t)tile * Z::TILE_WORDS);
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < nt; j++) {
        uint32_t *cv = smem_sg + j * HW, *c = cv + B::RING_WORDS, *io = tiles + (size_t)(tile0 + j) * Z::TILE_WORDS;
        for (int v = lane; v < (T + 1) * SS; v += 32) {
            const int i = v / SS, k = v - i * SS;
            io[(T - i) * SS + k] = c[v];
        }
        __syncwarp();
        for (int v = lane; v < NX * SS; v += 32)
            cv[v] = v < (T + 1) * SS ? io[v] : 0u;
        __syncwarp();
        fft_convert<S, SS, 32>(cv, scalpow, lane, [] { __syncwarp(); });
        for (int v = lane; v < NX * SS; v += 32)
            io[v] = cv[v];
    }
}

// The additive FFT of a tile's locators, a warp per ciphertext in turn, gridDim.y
// blocks a tile: flags
// flags[c * 2^(m-5) + w] = the zero test of elements 32w .. 32w + 31 in FFT
// position order.  Bound by the logic pipe; 13 KB a warp, twelve warps an SM.
template <int S>
__global__ void __launch_bounds__(FFT_WARPS * 32, 3) k_fft_tile(const uint32_t *__restrict__ tiles, uint32_t count,
                                                                const uint32_t *__restrict__ tw,
                                                                uint32_t *__restrict__ flags,
                                                                const StagedPiece *__restrict__ pieces)
{
    using Z = SgDims<S>;
    constexpr int SS = Z::SS, NX = Z::NX, NWD = Z::NWD, R = FftDims<S>::R;
    extern __shared__ __align__(16) uint32_t smem_sg[];
    uint32_t *cv = smem_sg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *fa = smem_sg + NX * SS + warp * FftDims<S>::FA_WORDS;
    const uint32_t *src = tiles + (size_t)blockIdx.x * Z::TILE_WORDS;
    for (int v = threadIdx.x; v < NX * SS; v += FFT_WARPS * 32)
        cv[v] = src[v];
    __syncthreads();
    const uint32_t c0 = 32 * blockIdx.x, n = pieces ? pieces[blockIdx.x].count : min(count - c0, 32u);
#pragma unroll 1
    for (int q = blockIdx.y * FFT_WARPS + warp; q < (int)n; q += FFT_WARPS * gridDim.y) {
        uint32_t z[R];
        fft_eval_one<S, SS>(cv, q, fa, tw, lane, z);
#pragma unroll
        for (int j = 0; j < R; j++)
            flags[(size_t)(c0 + q) * NWD + lane + 32 * j] = z[j];
    }
}

struct NetArgs {
    const uint32_t *flags;
    const uint32_t *bctl;
    uint32_t count;
    uint32_t *err;        // rows of nw words, or null
    uint16_t *weight;     // or null
    uint16_t *pos;        // rows of t + 1, or null
    StagedMixed mx;       // MIX: count is 32 * tiles, err / weight by ciphertext
};

// The support network of NC ciphertexts a warp: each layer's mask words are loaded
// once for all of them (they wait on memory, 25 layers in a row).
template <int S, int NC, bool MIX = false> __global__ void __launch_bounds__(NET_WARPS * 32) k_net_rows(NetArgs a)
{
    using F = FftDims<S>;
    constexpr int NWD = F::NWD, R = F::R;
    __shared__ uint32_t rows[NET_WARPS][NC * NWD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t c0 = ((uint64_t)blockIdx.x * NET_WARPS + warp) * NC;
    if (c0 >= a.count)
        return;
    int n = (int)(a.count - c0 < NC ? a.count - c0 : NC);
    const uint32_t *order = nullptr;
    if constexpr (MIX) {
        const StagedPiece t = a.mx.tiles[c0 / 32];
        const int left = (int)t.count - (int)(c0 % 32);
        n = left < NC ? left : NC;
        if (n <= 0)
            return;
        a.bctl = a.mx.keys[t.key].bctl;
        order = a.mx.order + t.first + c0 % 32;
    }
    uint32_t z[NC][R];
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < R; j++)
            z[i][j] = i < n ? a.flags[(c0 + i) * NWD + lane + 32 * j] : 0u;
    swap_network<S, NC>(z, a.bctl, lane);
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < R; j++)
            rows[warp][i * NWD + lane + 32 * j] = z[i][j];
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        uint32_t v[R];
#pragma unroll
        for (int j = 0; j < R; j++)
            v[j] = rows[warp][i * NWD + lane + 32 * j];  // this lane's own words
        const uint64_t c = MIX ? order[i] : c0 + i;
        const int cnt = root_output<S>(v, a.err ? a.err + (MIX ? a.mx.err_off[c] : c * F::NW) : nullptr,
                                       a.pos ? a.pos + c * (F::T + 1) : nullptr, nullptr, lane);
        if (lane == 0 && a.weight)
            a.weight[c] = (uint16_t)cnt;
    }
}

// Raises kernel `f`'s shared-memory limit once per device.
template <class K> cudaError_t allow_smem(K *f, size_t smem, bool (&given)[64])
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (given[dev & 63])
        return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    given[dev & 63] = e == cudaSuccess;
    return e;
}

}  // namespace

// Scratch words of a batch: tiles, then flags.
size_t staged_scratch_words(int set, size_t count)
{
    const size_t ntiles = (count + 31) / 32;
    return dispatch_set(set, [&]<int S>() -> size_t {
        return ntiles * SgDims<S>::TILE_WORDS + ntiles * 32 * SgDims<S>::NWD;
    });
}

cudaError_t launch_staged(const KeyDev &k, const uint8_t *d_cts, uint32_t count, uint32_t *d_scratch, uint32_t *d_err,
                          uint16_t *d_weight, uint16_t *d_pos, const FftPlanDev &plan, int num_sms,
                          bool many_parts, cudaStream_t s, LaunchCounter lc)
{
    if (count == 0)
        return cudaSuccess;
    return dispatch_set(k.set, [&]<int S>() -> cudaError_t {
        using Z = SgDims<S>;
        const uint32_t ntiles = (count + 31) / 32;
        uint32_t *tiles = d_scratch, *flags = tiles + (size_t)ntiles * Z::TILE_WORDS;
        // tiles per block: the whole batch in as few equal waves as possible
        const uint32_t sms = (uint32_t)num_sms;
        const int split = ntiles <= SYND_WARPS / 8 * sms ? 8 : ntiles <= SYND_WARPS / 4 * sms ? 4 : 1;
        const uint32_t most = sms * (SYND_WARPS / split), waves = (ntiles + most - 1) / most;
        const uint32_t bt = (ntiles + sms * waves - 1) / (sms * waves), blocks = (ntiles + bt - 1) / bt;
        const size_t synd_smem = 4 * (Z::ROW_WORDS + Z::COMB_WORDS) + (size_t)bt * 32 * Set<S>::CT + 16;
        const size_t synd_max = 4 * (Z::ROW_WORDS + Z::COMB_WORDS) + (size_t)SYND_WARPS * 32 * Set<S>::CT + 16;
        const size_t fft_smem = 4 * (size_t)(Z::NX * Z::SS + FFT_WARPS * FftDims<S>::FA_WORDS);
        static bool g0[64] = {}, g1[64] = {}, g2[64] = {}, g3[64] = {};
        cudaError_t e;
        if ((e = allow_smem(k_synd_table<S, 1>, synd_max, g0)) != cudaSuccess ||
            (e = allow_smem(k_synd_table<S, 4>, synd_max, g1)) != cudaSuccess ||
            (e = allow_smem(k_synd_table<S, 8>, synd_max, g3)) != cudaSuccess ||
            (e = allow_smem(k_fft_tile<S>, fft_smem, g2)) != cudaSuccess)
            return e;
        const uint32_t threads = bt * 32 * split;
        if (split == 8)
            k_synd_table<S, 8><<<blocks, threads, synd_smem, s>>>(k.tabd, d_cts, count, tiles, {});
        else if (split == 4)
            k_synd_table<S, 4><<<blocks, threads, synd_smem, s>>>(k.tabd, d_cts, count, tiles, {});
        else
            k_synd_table<S, 1><<<blocks, threads, synd_smem, s>>>(k.tabd, d_cts, count, tiles, {});
        // Warps a tile, by tiles an SM: enough that every scheduler has a warp, and two
        // to even out the schedulers when they would hold one or two; otherwise one,
        // which passes no barriers.  Whole call, t = 119, one / two / four warps: one
        // tile an SM 659 / 524 / 443 us, two 736 / 601 / 681, 2.5 769 / 852 / 886,
        // three 802 / 882 / 917, four 882 / 960 / 1,165, five 1,359 / 1,293 / 1,475; the
        // other sets alike (t = 64 at five 505 / 497 / 669).  37,888 ciphertexts, eight
        // an SM: 1,534 with one, 1,693 with two.
        const int bw = ntiles <= sms ? 4 : ntiles <= 2 * sms ? 2 : ntiles <= 4 * sms ? 1 : ntiles <= 6 * sms ? 2 : 1;
        const size_t bm_smem = 4 * (size_t)(Z::BM_WORDS + 2 * bw * 16);
        // Two tiles a warp where the SM holds at least two such warps a scheduler
        // (t = 64; with five or six of them an SM, t >= 119, 2^20 ciphertexts are
        // 0.5 to 6 % slower, with seven, t = 96, 1 %) and other parts fill the ends
        // of the coarser waves (100,000 ciphertexts in two parts 3 % slower,
        // 131,073 in three the same, 200,000 4 % faster, 2^20 5.6 %).
        bool pairs = false;
        if constexpr (Z::PAIRS) {
            pairs = many_parts;
            if (pairs)
                k_bm_pair<S><<<(ntiles + 1) / 2, 32, 8 * Z::PAIR_WORDS, s>>>(tiles, ntiles, count, plan.scalpow);
        }
        if (pairs)
            ;
        else if (bw == 4)
            k_bm_tile<S, 4><<<ntiles, 128, bm_smem, s>>>(tiles, count, plan.scalpow, sms, nullptr);
        else if (bw == 2)
            k_bm_tile<S, 2><<<ntiles, 64, bm_smem, s>>>(tiles, count, plan.scalpow, 2 * sms, nullptr);
        else
            k_bm_tile<S, 1><<<ntiles, 32, bm_smem, s>>>(tiles, count, plan.scalpow, 1, nullptr);
        // enough blocks for three an SM, up to a ciphertext a warp
        uint32_t parts = 1;
        while (parts < 32 / FFT_WARPS && ntiles * parts < 3 * sms)
            parts *= 2;
        k_fft_tile<S><<<dim3(ntiles, parts), FFT_WARPS * 32, fft_smem, s>>>(tiles, count, plan.tw, flags, nullptr);
        const NetArgs na{flags, k.bctl, count, d_err, d_weight, d_pos, {}};
        const uint32_t nc = count <= 64 * sms ? 1 : 4, per = NET_WARPS * nc;
        if (nc == 1)
            k_net_rows<S, 1><<<(count + per - 1) / per, NET_WARPS * 32, 0, s>>>(na);
        else
            k_net_rows<S, 4><<<(count + per - 1) / per, NET_WARPS * 32, 0, s>>>(na);
        lc.bump(4);
        return cudaGetLastError();
    });
}

cudaError_t launch_staged_mixed(int set, const StagedMixed &mx, uint32_t nblocks, uint32_t ntiles,
                                const uint8_t *d_cts, uint32_t *d_scratch, uint32_t *d_err, uint16_t *d_weight,
                                const FftPlanDev &plan, int num_sms, cudaStream_t s, LaunchCounter lc)
{
    if (ntiles == 0)
        return cudaSuccess;
    return dispatch_set(set, [&]<int S>() -> cudaError_t {
        using Z = SgDims<S>;
        constexpr uint32_t bt = staged_block_tiles;
        const uint32_t sms = (uint32_t)num_sms;
        uint32_t *tiles = d_scratch, *flags = tiles + (size_t)ntiles * Z::TILE_WORDS;
        constexpr size_t synd_smem = 4 * (Z::ROW_WORDS + Z::COMB_WORDS) + (size_t)bt * 32 * Set<S>::CT + 16;
        const size_t bm_smem = 4 * (size_t)(Z::BM_WORDS + 2 * 16);
        const size_t fft_smem = 4 * (size_t)(Z::NX * Z::SS + FFT_WARPS * FftDims<S>::FA_WORDS);
        static bool g0[64] = {}, g1[64] = {}, g2[64] = {};
        const bool split = nblocks < sms;  // more warps a tile, as for one key
        cudaError_t e;
        if ((e = allow_smem(k_synd_table<S, 1, true>, synd_smem, g0)) != cudaSuccess ||
            (e = allow_smem(k_synd_table<S, 2, true>, synd_smem, g1)) != cudaSuccess ||
            (e = allow_smem(k_fft_tile<S>, fft_smem, g2)) != cudaSuccess)
            return e;
        if (split)
            k_synd_table<S, 2, true><<<nblocks, bt * 64, synd_smem, s>>>(nullptr, d_cts, 0, tiles, mx);
        else
            k_synd_table<S, 1, true><<<nblocks, bt * 32, synd_smem, s>>>(nullptr, d_cts, 0, tiles, mx);
        k_bm_tile<S, 1><<<ntiles, 32, bm_smem, s>>>(tiles, 0, plan.scalpow, 1, mx.tiles);
        uint32_t parts = 1;
        while (parts < 32 / FFT_WARPS && ntiles * parts < 3 * sms)
            parts *= 2;
        k_fft_tile<S><<<dim3(ntiles, parts), FFT_WARPS * 32, fft_smem, s>>>(tiles, 0, plan.tw, flags, mx.tiles);
        const NetArgs na{flags, nullptr, 32 * ntiles, d_err, d_weight, nullptr, mx};
        k_net_rows<S, 4, true><<<(ntiles + NET_WARPS / 8 - 1) / (NET_WARPS / 8), NET_WARPS * 32, 0, s>>>(na);
        lc.bump(4);
        return cudaGetLastError();
    });
}

}  // namespace cmd

// Per-ciphertext decrypt kernels for small batches: no bitslicing across
// ciphertexts, each ciphertext with its own key and set.
//
// The other decrypt kernels run Berlekamp-Massey bitsliced across 32
// ciphertexts, so a tile of one costs what a tile of 32 does: 2t dependent
// steps of three 13 x 13-plane products each, with a warp's latency in every
// step (2.2 k cycles a step in k_tile_bm).  A small batch leaves the GPU idle
// meanwhile.  Here every ciphertext has its own warps and Berlekamp-Massey
// works on scalars, so a step is a few hundred cycles:
//
//  1. syndromes by the transposed additive FFT (latency.cu describes it): the
//     ciphertext bits through the key's support network in reverse, the key's
//     weights, D' butterfly levels over the 2^m-element bitsliced array, the
//     group parities, the transposed radix conversion;
//  2. scaled Berlekamp-Massey (bm.c:12-68, as in latency.cu): C in registers,
//     B in a shared ring whose rotation is the x*B shift, both loops bounded
//     by L.  Products are integer multiplies on operands with holes (gf.cuh),
//     the syndromes kept split into their four bit classes;
//  3. radix conversion of the locator, the additive-FFT root search and the
//     support network (fft_root.cuh), outputs.
//
// WPC warps share a ciphertext in a step.  Measured on a B200 (tile kernels ->
// these): one ciphertext of mceliece6960119 368 -> 78 us, 37 of 348864 187 ->
// 46 us, 1,184 of 6960119 388 -> 180 us; above about 24 ciphertexts an SM the
// tile kernels' bitsliced Berlekamp-Massey wins (4,736: 496 against 580 us).
// Bound by the latency of the serial Berlekamp-Massey chain up to one
// ciphertext an SM, by the multiply and logic pipes above.  Constant time as
// the other paths: no address or branch depends on the key or the error
// vector, except Berlekamp-Massey's trajectory of L.
#include <algorithm>

#include "fft_root.cuh"
#include "gf.cuh"
#include "internal.h"

namespace cmd {

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr int CT_WARPS = 4;              // warps per block
constexpr int CT_FA_WORDS = 13 * 256;    // FFT array, largest set
constexpr int CT_CV_WORDS = 256 / 2;     // u16 group sums, then locator constants
constexpr int CT_XB_WORDS = 2 * 256;     // cross-warp exchange of the network (WPC > 1)
// inside the FFT array while it is free (conversions and Berlekamp-Massey)
constexpr int CT_SS = 256;               // u32 sx[256] at 0, then uint4 split syndromes [2t]
constexpr int CT_RING = CT_SS + 4 * 256; // then the B ring [t + 2] (uint4 split values, or u32)
constexpr int CT_SHARE = CT_RING + 4 * 132;  // then the warps' shares, 2 x WPC uint2
static_assert(CT_SHARE + 2 * 2 * CT_WARPS <= CT_FA_WORDS, "Berlekamp-Massey data inside the FFT array");

enum Phase { ALL, SYND, BM, ROOT };

// Shared-memory words of one ciphertext's group.
template <Phase PH, int WPC> constexpr int ct_words()
{
    return PH == BM ? CT_SHARE + 2 * 2 * CT_WARPS : CT_FA_WORDS + CT_CV_WORDS + (WPC > 1 ? CT_XB_WORDS : 0);
}

// A field element's bits in four classes, positions = c (mod 4) (gf_mul_im).
struct Split {
    uint32_t c0, c1, c2, c3;
};
constexpr uint32_t K0 = 0x11111111u, K1 = K0 << 1, K2 = K0 << 2, K3 = K0 << 3;

// r | (p & k) as one lop3 (grouped otherwise by the compiler, seven for four).
__device__ __forceinline__ uint32_t pick(uint32_t r, uint32_t p, uint32_t k)
{
    uint32_t o;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(o) : "r"(p), "r"(k), "r"(r));
    return o;
}

__device__ __forceinline__ Split split4(uint32_t a) { return {a & K0, a & K1, a & K2, a & K3}; }

// Unreduced carry-less product (bits 0 .. 2m-2).
__device__ __forceinline__ uint32_t clmul_split(const Split &a, const Split &b)
{
    const uint32_t p0 = a.c0 * b.c0 + a.c1 * b.c3 + a.c2 * b.c2 + a.c3 * b.c1;
    const uint32_t p1 = a.c0 * b.c1 + a.c1 * b.c0 + a.c2 * b.c3 + a.c3 * b.c2;
    const uint32_t p2 = a.c0 * b.c2 + a.c1 * b.c1 + a.c2 * b.c0 + a.c3 * b.c3;
    const uint32_t p3 = a.c0 * b.c3 + a.c1 * b.c2 + a.c2 * b.c1 + a.c3 * b.c0;
    return pick(pick(pick(p0 & K0, p1, K1), p2, K2), p3, K3);
}

// The Taylor steps of one radix-conversion depth d on scalar entries sx[x],
// by one warp.  A thread takes the same two quads at every step, so that the
// two dependent XORs of a step need no barrier between them.
template <int D, bool TRANSPOSED> __device__ __forceinline__ void taylor_scalar(uint32_t *sx, int d, int lane)
{
    constexpr int NX = 1 << D;
#pragma unroll 1
    for (int s = 2; s <= D - d; s++) {
        const int kb = TRANSPOSED ? s : D - d + 2 - s;
        const int Q = 1 << (kb - 2);
#pragma unroll
        for (int u = lane; u < NX / 4; u += 32) {
            const int sub = u & ((1 << d) - 1), rest = u >> d;
            const int i = (rest >> (kb - 2)) * 4 * Q + (rest & (Q - 1));
            uint32_t *x = sx + (i << d) + sub;
            const int q = Q << d;
            const uint32_t x1 = x[q], x2 = x[2 * q], x3 = x[3 * q];
            if (TRANSPOSED) {  // third ^= second; fourth ^= third
                x[2 * q] = x2 ^ x1;
                x[3 * q] = x3 ^ x2 ^ x1;
            } else {  // third ^= fourth; second ^= third
                x[2 * q] = x2 ^ x3;
                x[q] = x1 ^ x2 ^ x3;
            }
        }
        __syncwarp();
    }
}

// The transposed radix conversion (fft_convert_t) of scalar entries sx[x]:
// Taylor steps by the first warp, scalings by the whole group.
template <int S, int WPC>
__device__ __forceinline__ void convert_t_scalar(uint32_t *sx, const uint16_t *__restrict__ scalpow, int tid)
{
    constexpr int M = Set<S>::M, D = synd_depth(Set<S>::T), NX = 1 << D, NT = 32 * WPC, PER = (NX + NT - 1) / NT;
#pragma unroll 1
    for (int d = D - 1; d >= 0; d--) {
        uint32_t c[PER];
#pragma unroll
        for (int k = 0; k < PER; k++)
            c[k] = __ldg(scalpow + d * 256 + ((tid + NT * k) >> d));
        if (tid < 32)
            taylor_scalar<D, true>(sx, d, tid);
        group_sync<WPC>();
        if (d > 0) {
#pragma unroll
            for (int k = 0; k < PER; k++)
                if (tid + NT * k < NX)
                    sx[tid + NT * k] = gf_mul_im<M>(sx[tid + NT * k], c[k]);
            group_sync<WPC>();
        }
    }
}

// The radix conversion (fft_convert) of scalar entries sx[x].
template <int S, int WPC>
__device__ __forceinline__ void convert_scalar(uint32_t *sx, const uint16_t *__restrict__ scalpow, int tid)
{
    using F = FftDims<S>;
    constexpr int M = F::M, D = F::D, NX = F::NX, NT = 32 * WPC, PER = (NX + NT - 1) / NT;
#pragma unroll 1
    for (int d = 0; d < D; d++) {
        uint32_t c[PER];
#pragma unroll
        for (int k = 0; k < PER; k++)  // depth d + 1's scalings
            c[k] = d + 1 < D ? __ldg(scalpow + (d + 1) * 256 + ((tid + NT * k) >> (d + 1))) : 0u;
        if (tid < 32)
            taylor_scalar<D, false>(sx, d, tid);
        group_sync<WPC>();
        if (d + 1 < D) {
#pragma unroll
            for (int k = 0; k < PER; k++)
                if (tid + NT * k < NX)
                    sx[tid + NT * k] = gf_mul_im<M>(sx[tid + NT * k], c[k]);
            group_sync<WPC>();
        }
    }
}

// One step of the one-warp Berlekamp-Massey with the first NA groups of 32
// coefficients active (straight-line code, so the groups' products overlap).
template <int S, int NA, int NJ>
__device__ __forceinline__ void bm_step(const uint4 *ss, uint4 *ring, uint32_t (&C)[NJ], Split &b, int &L, int &off,
                                        int N, int lane)
{
    constexpr int M = Set<S>::M, T = Set<S>::T, R = T + 2;
    uint32_t q[NA], pd = 0;
    uint4 bv[NA];
    Split c[NA];
#pragma unroll
    for (int j = 0; j < NA; j++) {
        const int i = lane + 32 * j;
        int slot = i + off;
        slot = slot >= R ? slot - R : slot;
        bv[j] = i <= T ? ring[slot] : make_uint4(0, 0, 0, 0);
        const uint4 s = ss[max(N - i, 0)];  // C_i = 0 where N < i
        c[j] = split4(C[j]);
        pd ^= clmul_split(c[j], Split{s.x, s.y, s.z, s.w});
        q[j] = clmul_split(c[j], b);
    }
    const uint32_t d = __reduce_xor_sync(FULL, gf_reduce<M>(pd));
    const bool swap = d != 0 && N >= 2 * L;
    const Split ds = split4(d);
    __syncwarp();  // B is read before the swap overwrites it
    if (swap) {    // B <- C, zero above the active groups
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int i = lane + 32 * j;
            int slot = i + off;
            slot = slot >= R ? slot - R : slot;
            if (i <= T)
                ring[slot] = j < NA ? make_uint4(c[j < NA ? j : 0].c0, c[j < NA ? j : 0].c1, c[j < NA ? j : 0].c2,
                                                 c[j < NA ? j : 0].c3)
                                    : make_uint4(0, 0, 0, 0);
        }
    }
#pragma unroll
    for (int j = 0; j < NA; j++)
        C[j] = gf_reduce<M>(q[j] ^ clmul_split(Split{bv[j].x, bv[j].y, bv[j].z, bv[j].w}, ds));
    if (swap) {
        L = N + 1 - L;
        b = ds;
    }
    // the slot that becomes coefficient 0 of x*B
    off = off == 0 ? R - 1 : off - 1;
    if (lane == 0)
        ring[off] = make_uint4(0, 0, 0, 0);
    __syncwarp();
}

// One warp: scaled Berlekamp-Massey on the syndromes ss[0 .. 2t) (split);
// leaves sx[t - i] = C_i, zero above t.
template <int S> __device__ __forceinline__ void bm_warp(const uint4 *ss, uint4 *ring, uint32_t *sx, int lane)
{
    using F = FftDims<S>;
    constexpr int T = F::T, NX = F::NX, NJ = (T + 32) / 32, R = T + 2;
    for (int v = lane; v < R; v += 32)
        ring[v] = make_uint4(v == 1, 0, 0, 0);  // B = x, split
    uint32_t C[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++)
        C[j] = lane + 32 * j == 0;
    Split b = split4(1);
    int L = 0, off = 0;  // ring slot of coefficient i at step N: i + off, off = -N mod R
    __syncwarp();
#pragma unroll 1
    for (int N = 0; N < 2 * T; N++) {
        // C is zero above L, and above the larger of L and N + 1 - L after
        // the step, whether or not the step swaps
        const int na = min(max(L, N + 1 - L), T) / 32 + 1;
        if (na == 1)
            bm_step<S, 1, NJ>(ss, ring, C, b, L, off, N, lane);
        else if (na == 2)
            bm_step<S, 2, NJ>(ss, ring, C, b, L, off, N, lane);
        else if (NJ <= 3 || na == 3)
            bm_step<S, NJ < 3 ? NJ : 3, NJ>(ss, ring, C, b, L, off, N, lane);
        else if (NJ <= 4 || na == 4)
            bm_step<S, NJ < 4 ? NJ : 4, NJ>(ss, ring, C, b, L, off, N, lane);
        else
            bm_step<S, NJ, NJ>(ss, ring, C, b, L, off, N, lane);
    }
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int i = lane + 32 * j;
        if (i <= T)
            sx[T - i] = C[j];
    }
    for (int x = T + 1 + lane; x < NX; x += 32)
        sx[x] = 0;
}

// The same by WPC warps, thread tid owning coefficients tid, tid + 32 WPC, ...,
// for the shortest time of one ciphertext.  The discrepancy is looked ahead:
//   d_{N+1} = sum_i (b C_i + d_N B_i) S_{N+1-i} = b <C, S_{N+1}> + d_N <B, S_{N+1}>,
// so both sums over the coefficients, their reductions and the exchange
// between the warps run beside step N's update instead of after it, and the
// chain from one discrepancy to the next is one scalar product pair.  That is
// a fourth product per coefficient, on pipes that one ciphertext leaves idle.
template <int S, int WPC>
__device__ __forceinline__ void bm_group(const uint4 *ss, uint32_t *ring, uint2 *share, uint32_t *sx, int tid)
{
    using F = FftDims<S>;
    constexpr int M = F::M, T = F::T, NX = F::NX, NT = 32 * WPC, NJ = (T + NT) / NT, R = T + 2;
    for (int v = tid; v < R; v += NT)
        ring[v] = v == 1;  // B = x
    uint32_t C[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++)
        C[j] = tid + NT * j == 0;
    if (tid < WPC)  // d_0 = S_0 = b * S_0 + d * 0
        share[tid] = make_uint2(tid == 0 ? ss[0].x | ss[0].y | ss[0].z | ss[0].w : 0u, 0u);
    Split b = split4(1), bp = b, dp = split4(0);  // b; b and d of the step before
    int L = 0, off = 0;
    group_sync<WPC>();
#pragma unroll 1
    for (int N = 0; N < 2 * T; N++) {
        const int hi = min(max(L, N + 1 - L), T);  // bounds deg C, deg B and deg of the new C
        uint2 *sh = share + (N & 1) * WPC;  // rewritten two barriers later
        uint32_t es = 0, fs = 0;
#pragma unroll
        for (int w = 0; w < WPC; w++) {
            const uint2 v = sh[w];
            es ^= v.x;
            fs ^= v.y;
        }
        uint32_t pe = 0, pf = 0, B[NJ], q[NJ];
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int i = tid + NT * j;
            int slot = i + off;
            slot = slot >= R ? slot - R : slot;
            B[j] = i <= T ? ring[slot] : 0u;
            q[j] = 0;
            if (j == 0 || NT * j <= hi) {
                const uint4 sv = ss[min(max(N + 1 - i, 0), 2 * T - 1)];  // C_i = B_i = 0 where N + 1 < i
                const Split s{sv.x, sv.y, sv.z, sv.w}, c = split4(C[j]);
                pe ^= clmul_split(c, s);
                pf ^= clmul_split(split4(B[j]), s);
                q[j] = clmul_split(c, b);
            }
        }
        const uint32_t d = gf_reduce<M>(clmul_split(split4(es), bp) ^ clmul_split(split4(fs), dp));
        const uint32_t e = __reduce_xor_sync(FULL, gf_reduce<M>(pe)), f = __reduce_xor_sync(FULL, gf_reduce<M>(pf));
        if ((tid & 31) == 0)
            share[(~N & 1) * WPC + (tid >> 5)] = make_uint2(e, f);
        const bool swap = d != 0 && N >= 2 * L;
        const Split ds = split4(d);
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int i = tid + NT * j;
            int slot = i + off;
            slot = slot >= R ? slot - R : slot;
            if (i <= T)
                ring[slot] = swap ? C[j] : B[j];
            if (j == 0 || NT * j <= hi)
                C[j] = i <= T ? gf_reduce<M>(q[j] ^ clmul_split(split4(B[j]), ds)) : 0u;
        }
        bp = b;
        dp = ds;
        if (swap) {
            L = N + 1 - L;
            b = ds;
        }
        off = off == 0 ? R - 1 : off - 1;
        if (tid == 0)
            ring[off] = 0;  // coefficient 0 of x*B
        group_sync<WPC>();
    }
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int i = tid + NT * j;
        if (i <= T)
            sx[T - i] = C[j];
    }
    for (int x = T + 1 + tid; x < NX; x += NT)
        sx[x] = 0;
}

// Step 1: the syndromes of one ciphertext, sx[0 .. 2t).
template <int S, int WPC>
__device__ __forceinline__ void synd_phase(const LatItem &it, const uint8_t *__restrict__ cts, const FftPlanDev &pl,
                                           uint32_t *smem, int tid)
{
    using F = FftDims<S>;
    using P = Set<S>;
    constexpr int M = F::M, T = F::T, NWD = F::NWD, NT = 32 * WPC, R = NWD / NT, CTW = P::CTW;
    constexpr int DS = synd_depth(T);
    static_assert(DS == M - 5, "one word per group of the transposed FFT");
    static_assert(R >= 1 && F::FA_WORDS <= CT_FA_WORDS, "work split");
    uint32_t *fa = smem, *sx = smem;
    uint16_t *cv = reinterpret_cast<uint16_t *>(smem + CT_FA_WORDS);
    uint32_t *xb = smem + CT_FA_WORDS + CT_CV_WORDS;
    int half = 0;
    const uint32_t *__restrict__ tw = pl.tw;
    const uint8_t *c = cts + it.ct_off;
    uint32_t z[R];
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int w = tid + NT * j;
        uint32_t v = 0;
        if (w < CTW) {
#pragma unroll
            for (int b = 0; b < 4; b++)
                if (4 * w + b < P::CT)
                    v |= (uint32_t)__ldg(c + 4 * w + b) << (8 * b);
        }
        z[j] = v;
    }
#pragma unroll
    for (int l = 2 * M - 2; l >= 0; l--)
        swap_layer<S, WPC>(z, it.bctl, l, tid, xb, &half);
    if constexpr (R == 1) {  // depth 0 pairs words of different threads
        xb[half * NWD + tid] = z[0];
        group_sync<WPC>();
    }
#pragma unroll
    for (int j = 0; j < (R + 1) / 2; j++) {
        const int wa = tid + NT * j, wb = wa + NWD / 2;
        if (R == 1 && wa >= NWD / 2)
            break;
        const uint32_t za = R == 1 ? xb[half * NWD + wa] : z[j];
        const uint32_t zb = R == 1 ? xb[half * NWD + wb] : z[R > 1 ? j + R / 2 : 0];
        uint32_t A[M], B[M], G[M], p[2 * M - 1];
#pragma unroll
        for (int k = 0; k < M; k++) {
            B[k] = zb & __ldg(it.wfft + k * NWD + wb);
            A[k] = (za & __ldg(it.wfft + k * NWD + wa)) ^ B[k];
            G[k] = __ldg(tw + wa + k * NWD);
        }
#pragma unroll
        for (int k = 0; k < 2 * M - 1; k++)
            p[k] = 0;
        bs_mul_acc<M>(p, G, A);
        bs_reduce<M>(p);
        const int pa = fa_word(wa), pb = fa_word(wb);
#pragma unroll
        for (int k = 0; k < M; k++) {
            fa[k * NWD + pa] = A[k];
            fa[k * NWD + pb] = B[k] ^ p[k];
        }
    }
    group_sync<WPC>();
#pragma unroll 1
    for (int d = 1; d < DS; d++) {
        const int sbit = M - d - 6, Sw = 1 << sbit;
        const uint32_t *twd = tw + tw_offset<M>(d);
#pragma unroll 1
        for (int P2 = tid; P2 < NWD / 2; P2 += NT) {
            const int wa = ((P2 >> sbit) << (sbit + 1)) | (P2 & (Sw - 1));
            const uint32_t *g = twd + (P2 & (Sw - 1));
            const int pa = fa_word(wa), pb = fa_word(wa + Sw);
            uint32_t A[M], B[M], G[M], p[2 * M - 1];
#pragma unroll
            for (int k = 0; k < M; k++) {
                B[k] = fa[k * NWD + pb];
                A[k] = fa[k * NWD + pa] ^ B[k];
                G[k] = __ldg(g + k * NWD);
            }
#pragma unroll
            for (int k = 0; k < 2 * M - 1; k++)
                p[k] = 0;
            bs_mul_acc<M>(p, G, A);
            bs_reduce<M>(p);
            if (d < DS - 1) {
#pragma unroll
                for (int k = 0; k < M; k++) {
                    fa[k * NWD + pa] = A[k];
                    fa[k * NWD + pb] = B[k] ^ p[k];
                }
            } else {  // each word is a group: its parities are a group sum
                uint32_t va = 0, vb = 0;
#pragma unroll
                for (int k = 0; k < M; k++) {
                    va |= (uint32_t)(__popc(A[k]) & 1) << k;
                    vb |= (uint32_t)(__popc(B[k] ^ p[k]) & 1) << k;
                }
                cv[__brev((uint32_t)wa) >> (32 - DS)] = (uint16_t)va;
                cv[__brev((uint32_t)(wa + Sw)) >> (32 - DS)] = (uint16_t)vb;
            }
        }
        group_sync<WPC>();
    }
    for (int x = tid; x < (1 << DS); x += NT)
        sx[x] = cv[x];
    group_sync<WPC>();
    convert_t_scalar<S, WPC>(sx, pl.scalpow, tid);
}

// Step 2: from the syndromes sx[0 .. 2t) to the reversed locator sx[0 .. 2^D).
template <int S, int WPC> __device__ __forceinline__ void bm_phase(uint32_t *smem, int tid)
{
    constexpr int T = Set<S>::T;
    uint32_t *sx = smem;
    uint4 *ss = reinterpret_cast<uint4 *>(smem + CT_SS);
    for (int x = tid; x < 2 * T; x += 32 * WPC) {
        const Split v = split4(sx[x]);
        ss[x] = make_uint4(v.c0, v.c1, v.c2, v.c3);
    }
    group_sync<WPC>();
    if constexpr (WPC == 1)
        bm_warp<S>(ss, reinterpret_cast<uint4 *>(smem + CT_RING), sx, tid);
    else
        bm_group<S, WPC>(ss, smem + CT_RING, reinterpret_cast<uint2 *>(smem + CT_SHARE), sx, tid);
    group_sync<WPC>();
}

// Step 3: from the reversed locator sx[0 .. 2^D) to the outputs.
template <int S, int WPC>
__device__ __forceinline__ void root_phase(const LatItem &it, uint32_t *err, uint16_t *weight, uint16_t *pos,
                                           const FftPlanDev &pl, uint32_t *smem, int tid)
{
    using F = FftDims<S>;
    constexpr int M = F::M, D = F::D, NWD = F::NWD, NT = 32 * WPC, R = NWD / NT;
    uint32_t *fa = smem, *sx = smem;
    uint16_t *cv = reinterpret_cast<uint16_t *>(smem + CT_FA_WORDS);
    uint32_t *xb = smem + CT_FA_WORDS + CT_CV_WORDS;
    int half = 0;
    const uint32_t *__restrict__ tw = pl.tw;
    uint32_t z[R];
    convert_scalar<S, WPC>(sx, pl.scalpow, tid);
    for (int x = tid; x < F::NX; x += NT)
        cv[x] = (uint16_t)sx[x];
    group_sync<WPC>();
#pragma unroll 1
    for (int d = D - 1; d >= 1; d--) {
        const int sbit = M - d - 6, Sw = 1 << sbit;
        const uint32_t *twd = tw + tw_offset<M>(d);
#pragma unroll 1
        for (int P2 = tid; P2 < NWD / 2; P2 += NT) {
            const int wa = ((P2 >> sbit) << (sbit + 1)) | (P2 & (Sw - 1));
            const uint32_t *g = twd + (P2 & (Sw - 1));
            const int pa = fa_word(wa), pb = fa_word(wa + Sw);
            uint32_t A[M], B[M], G[M], p[2 * M - 1];
            if (d == D - 1) {  // both operands are depth-D constants
                const uint32_t ca = cv[__brev((uint32_t)(wa >> sbit)) >> (32 - D)];
                const uint32_t cb = cv[__brev((uint32_t)((wa + Sw) >> sbit)) >> (32 - D)];
#pragma unroll
                for (int k = 0; k < M; k++) {
                    A[k] = (uint32_t)((int32_t)(ca << (31 - k)) >> 31);
                    B[k] = (uint32_t)((int32_t)(cb << (31 - k)) >> 31);
                }
            } else {
#pragma unroll
                for (int k = 0; k < M; k++) {
                    A[k] = fa[k * NWD + pa];
                    B[k] = fa[k * NWD + pb];
                }
            }
#pragma unroll
            for (int k = 0; k < M; k++)
                G[k] = __ldg(g + k * NWD);
#pragma unroll
            for (int k = 0; k < 2 * M - 1; k++)
                p[k] = 0;
            bs_mul_acc<M>(p, G, B);
            bs_reduce<M>(p);
#pragma unroll
            for (int k = 0; k < M; k++) {
                const uint32_t na = A[k] ^ p[k];
                fa[k * NWD + pa] = na;
                fa[k * NWD + pb] = na ^ B[k];
            }
        }
        group_sync<WPC>();
    }
#pragma unroll
    for (int j = 0; j < (R + 1) / 2; j++) {
        const int wa = tid + NT * j, wb = wa + NWD / 2;
        if (R == 1 && wa >= NWD / 2)
            break;
        const int pa = fa_word(wa), pb = fa_word(wb);
        uint32_t A[M], B[M], G[M], p[2 * M - 1];
#pragma unroll
        for (int k = 0; k < M; k++) {
            A[k] = fa[k * NWD + pa];
            B[k] = fa[k * NWD + pb];
            G[k] = __ldg(tw + wa + k * NWD);
        }
#pragma unroll
        for (int k = 0; k < 2 * M - 1; k++)
            p[k] = 0;
        bs_mul_acc<M>(p, G, B);
        bs_reduce<M>(p);
        uint32_t anya = 0, anyb = 0;
#pragma unroll
        for (int k = 0; k < M; k++) {
            const uint32_t na = A[k] ^ p[k];
            anya |= na;
            anyb |= na ^ B[k];
        }
        if (R == 1) {
            xb[half * NWD + wa] = ~anya;
            xb[half * NWD + wb] = ~anyb;
        } else {
            z[j] = ~anya;
            z[R > 1 ? j + R / 2 : 0] = ~anyb;
        }
    }
    if constexpr (R == 1) {
        group_sync<WPC>();
        z[0] = xb[half * NWD + tid];
        half ^= 1;
    }
#pragma unroll
    for (int l = 0; l < 2 * M - 1; l++)
        swap_layer<S, WPC>(z, it.bctl, l, tid, xb, &half);
    uint32_t *erow = err && !it.row ? err + it.err_off : nullptr;
    int cnt;
    if constexpr (WPC == 1) {
        cnt = root_output<S>(z, erow, pos, it.row, tid);
    } else {
#pragma unroll
        for (int j = 0; j < R; j++)
            xb[half * NWD + tid + NT * j] = z[j];
        group_sync<WPC>();
        if (tid >= 32)
            return;
        uint32_t v[F::R];
#pragma unroll
        for (int j = 0; j < F::R; j++)
            v[j] = xb[half * NWD + tid + 32 * j];
        cnt = root_output<S>(v, erow, pos, it.row, tid);
    }
    // rows stored in host memory are visible before anything the stream
    // writes after this kernel
    if (it.row)
        __threadfence_system();
    if (tid == 0 && weight)
        *weight = (uint16_t)cnt;
}

struct CtArgs {
    const LatItem *items;  // or null: slots of one key (key0), rows back to back
    LatItem key0;
    uint32_t nslots;
    const uint8_t *cts;
    uint16_t *mid;         // three launches: 256 u16 per slot, syndromes, then the locator
    uint32_t *err;         // may be null
    uint16_t *weight;      // indexed by slot; may be null
    uint16_t *pos;         // rows of t + 1 by slot; may be null
    FftPlans plans;
};

// The slot of this thread's group, or false when the group has none (the
// whole group leaves: barriers are the group's).
template <int WPC> __device__ __forceinline__ bool take_slot(const CtArgs &a, uint32_t &slot, LatItem &it)
{
    slot = blockIdx.x * (CT_WARPS / WPC) + threadIdx.x / (32 * WPC);
    if (slot >= a.nslots)
        return false;
    if (a.items) {
        it = a.items[slot];
        return it.set >= 0;
    }
    it = a.key0;
    const SetInfo si = set_info(it.set);
    it.ct_off = slot * (uint32_t)si.ct;
    it.err_off = slot * (uint32_t)si.nw;
    return true;
}

template <class F> __device__ __forceinline__ void for_set(int set, F &&f)
{
    switch (set) {
    case S348864: f.template operator()<S348864>(); break;
    case S460896: f.template operator()<S460896>(); break;
    case S6688128: f.template operator()<S6688128>(); break;
    case S6960119: f.template operator()<S6960119>(); break;
    default: f.template operator()<S8192128>(); break;
    }
}

template <Phase PH, int WPC> __global__ void __launch_bounds__(CT_WARPS * 32, 4) k_ct(CtArgs a)
{
    extern __shared__ __align__(16) uint32_t smem_ct[];
    uint32_t slot;
    LatItem it;
    if (!take_slot<WPC>(a, slot, it))
        return;
    const int tid = threadIdx.x % (32 * WPC);
    uint32_t *smem = smem_ct + threadIdx.x / (32 * WPC) * ct_words<PH, WPC>();
    for_set(it.set, [&]<int S>() {
        uint16_t *mid = a.mid + (size_t)slot * 256;
        if (PH == ALL || PH == SYND)
            synd_phase<S, WPC>(it, a.cts, a.plans.p[S], smem, tid);
        if (PH == SYND)
            for (int x = tid; x < 2 * Set<S>::T; x += 32 * WPC)
                mid[x] = (uint16_t)smem[x];
        if (PH == BM)
            for (int x = tid; x < 2 * Set<S>::T; x += 32 * WPC)
                smem[x] = mid[x];
        if (PH == BM)
            group_sync<WPC>();
        if (PH == ALL || PH == BM)
            bm_phase<S, WPC>(smem, tid);
        if (PH == BM)
            for (int x = tid; x < FftDims<S>::NX; x += 32 * WPC)
                mid[x] = (uint16_t)smem[x];
        if (PH == ROOT)
            for (int x = tid; x < FftDims<S>::NX; x += 32 * WPC)
                smem[x] = mid[x];
        if (PH == ROOT)
            group_sync<WPC>();
        if (PH == ALL || PH == ROOT)
            root_phase<S, WPC>(it, a.err, a.weight ? a.weight + slot : nullptr,
                               a.pos ? a.pos + (size_t)slot * (Set<S>::T + 1) : nullptr, a.plans.p[S], smem, tid);
    });
}

template <Phase PH, int WPC> cudaError_t launch_phase(const CtArgs &a, cudaStream_t s, LaunchCounter lc)
{
    constexpr uint32_t CPB = CT_WARPS / WPC;
    constexpr size_t smem = CPB * ct_words<PH, WPC>() * 4;
    static bool given[64] = {};  // per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!given[dev & 63]) {
        cudaError_t e = cudaFuncSetAttribute(k_ct<PH, WPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_ct<PH, WPC>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess)
            return e;
        given[dev & 63] = true;
    }
    k_ct<PH, WPC><<<(a.nslots + CPB - 1) / CPB, CT_WARPS * 32, smem, s>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        lc.bump();
    return e;
}

// One launch, or the three steps apart, by the number of ciphertexts:
//  - up to CT_ONE_LAUNCH: one launch, four warps a ciphertext in every step
//    (one mceliece6960119 ciphertext 79 us against 88 us in three launches);
//  - while each has an SM to itself: three launches, four warps a ciphertext
//    (148: 91 us against 103 us with one warp in Berlekamp-Massey);
//  - above: one warp in Berlekamp-Massey, which issues 3/4 of the products and
//    no barriers (592: 120 us against 211 us; 1,184: 178 against 385 us).
//    The FFT steps keep four warps (592: 120 us against 132 us with one).
cudaError_t launch(const CtArgs &a, uint32_t live, int num_sms, cudaStream_t s, LaunchCounter lc)
{
    if (a.nslots == 0)
        return cudaSuccess;
    if (live <= CT_ONE_LAUNCH)
        return launch_phase<ALL, 4>(a, s, lc);
    cudaError_t e = launch_phase<SYND, 4>(a, s, lc);
    if (e == cudaSuccess)
        e = live <= (uint32_t)num_sms ? launch_phase<BM, 4>(a, s, lc) : launch_phase<BM, 1>(a, s, lc);
    if (e == cudaSuccess)
        e = launch_phase<ROOT, 4>(a, s, lc);
    return e;
}

}  // namespace

cudaError_t launch_ct_items(const LatItem *d_items, const uint8_t *d_cts, uint32_t nslots, uint32_t live,
                            uint16_t *d_mid, uint32_t *d_err, uint16_t *d_weight, uint16_t *d_pos,
                            const FftPlans &plans, int num_sms, cudaStream_t s, LaunchCounter lc)
{
    return launch(CtArgs{d_items, LatItem{}, nslots, d_cts, d_mid, d_err, d_weight, d_pos, plans}, live, num_sms, s,
                  lc);
}

cudaError_t launch_ct_one(const KeyDev &k, const uint8_t *d_cts, uint32_t count, uint32_t *d_err, uint16_t *d_weight,
                          uint16_t *d_pos, const FftPlans &plans, cudaStream_t s, LaunchCounter lc)
{
    const LatItem key{k.wfft, k.bctl, 0, 0, k.set, 0, nullptr};
    return launch(CtArgs{nullptr, key, count, d_cts, nullptr, d_err, d_weight, d_pos, plans}, count, 0, s, lc);
}

}  // namespace cmd

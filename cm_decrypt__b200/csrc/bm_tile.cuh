// Berlekamp-Massey (bm.c:12-68) bitsliced across the 32 ciphertexts of a tile:
// word bit q belongs to ciphertext q, lane l owns locator coefficients l, l + 32,
// ...  Coefficients, syndromes and B are rows of SS words in shared memory (SS = m
// made odd, so that lanes' rows meet no bank conflict; for m = 12 the 12-word rows
// of neighbouring lanes met four ways).
//
// The update is the scaled form C <- b*C + d*x*B instead of bm()'s C <- C +
// (d/b)*x*B: same decisions (d != 0, N >= 2L), same truncation, and by induction
// the result is lambda times bm()'s locator with lambda a product of nonzero b
// values -- the same roots, so the same flagged positions, with no inversion
// chain per step.  deg C <= L for every ciphertext, so only coefficients up to
// the tile's largest L take part (about half the slots of the reference loop
// bounds for weight-t errors, where L ~ N/2).  B lives in a ring of t + 2 rows
// whose rotation is the x*B shift.
//
// Bound by the logic pipe, so the products are what counts: one-level Karatsuba
// (KAcc) with b's and d's half sums formed once a step, b*C and d*B sharing one
// combination and reduction, and the next discrepancy's products taken on the
// new coefficient while it is in registers, all of a lane's terms sharing one
// combination.  In the fused kernel, against two passes over the coefficients
// with schoolbook products: 65,536 mceliece6960119 ciphertexts 3,125 -> 3,057 us,
// one tile an SM (9,472 ciphertexts in all) 1,173 -> 1,112 us.
#pragma once
#include "gf.cuh"
#include "params.h"

namespace cmd {

template <int S> struct BmDims {
    static constexpr int M = Set<S>::M, T = Set<S>::T, SS = M | 1, R = T + 2;
    static constexpr int SYN_WORDS = 2 * T * SS, RING_WORDS = R * SS, C_WORDS = (T + 1) * SS;
};

// W warps (thread tid < 32 W of them): syndromes -> locator coefficients C (rows
// of SS words); ntile: ciphertexts of the tile (the others' syndromes are zero).
//
// W = 1: the warp alone.  W > 1: groups of 32 coefficients go round the warps,
// which meet once a step (named barrier 1) to add their shares of the
// discrepancy (share: 2 W rows of 16 words); for batches that leave schedulers
// without a warp.  The first groups are active longest, so warp (W - turn) % W
// takes the first one: callers vary `turn` between the tiles of an SM.
//
// PAIR: a warp for two tiles, 16 lanes each, groups of 16 coefficients (syn, ring,
// cm, gsyn and ntile are then those of the lane's own tile; both tiles' arrays are
// the same distance apart, 16 mod 32 words, so that the halves' rows meet no bank
// conflict).  The loops are bounded by the larger L of the two, nearly always
// the same.  L grows from 0 to t, so that a tile takes 1.3 passes of 32 lanes a step
// instead of 1.5 (t = 64; t = 119: 2.2 instead of 2.5), and the work of a step
// outside the loop serves both tiles; but half the warps are left to hide its
// latency.
//
// The syndromes are either all in shared memory (syn, gsyn null) or in global
// memory (gsyn), one row a step coming into syn as a ring of t + 2 rows: step N
// multiplies rows N + 1 - L .. N + 1 only, and L stops at t.  The ring takes a
// quarter off a tile's shared memory.
template <int S, bool GLOBAL_SYN = false, int W = 1, bool PAIR = false>
__device__ __forceinline__ void bm_tile(uint32_t *syn, uint32_t *ring, uint32_t *cm, int ntile, int tid,
                                        const uint32_t *gsyn = nullptr, uint32_t *share = nullptr, int turn = 0)
{
    using Z = BmDims<S>;
    static_assert(W == 1 || !PAIR, "a pair of tiles: one warp");
    constexpr int M = Z::M, T = Z::T, SS = Z::SS, R = Z::R, H = KAcc<M>::H, NT = PAIR ? 16 : 32 * W;
    constexpr int NQ = PAIR ? 2 : 1;  // ciphertexts whose L a lane keeps: lane, lane + 16 of its tile
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const int lane = tid & 31, warp = tid >> 5;
    const bool upper = PAIR && lane >= 16;
    if (PAIR)
        tid &= 15;
    const int first = W == 1 ? tid : (tid + 32 * turn) % NT;  // this lane's first coefficient
    auto sync = [] {
        if constexpr (W == 1)
            __syncwarp();
        else
            asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
    };
    for (int v = tid; v < Z::C_WORDS; v += NT)
        cm[v] = v == 0 ? FULL : 0u;  // C = 1
    for (int v = tid; v < Z::RING_WORDS; v += NT)
        ring[v] = v == SS ? FULL : 0u;  // B = x
    if constexpr (GLOBAL_SYN) {
        for (int v = tid; v < 2 * SS; v += NT)
            syn[v] = gsyn[v];
        sync();
    }
    uint32_t b[M], p[2 * M - 1];  // p: this lane's share of the discrepancy
#pragma unroll
    for (int k = 0; k < M; k++) {
        b[k] = k == 0 ? FULL : 0u;      // b = 1
        p[k] = tid == 0 ? syn[k] : 0u;  // d_0 = C_0 S_0 (any one lane)
    }
    int Lq[NQ] = {}, Bd[NQ], Bmax = 1;  // L and a bound on deg B of the lane's ciphertexts; the latter's largest
#pragma unroll
    for (int h = 0; h < NQ; h++)
        Bd[h] = 1;
    if (W == 1)
        sync();
#pragma unroll 1
    for (int N = 0; N < 2 * T; N++) {
        uint32_t row = 0;
        if (GLOBAL_SYN && tid < SS && N + 2 < 2 * T)
            row = gsyn[(N + 2) * SS + tid];
        uint32_t d[M], mne = 0;
        if (PAIR && upper) {
#pragma unroll
            for (int k = 0; k < M; k++)
                d[k] = __reduce_xor_sync(0xFFFF0000u, p[k]);
        } else {
#pragma unroll
            for (int k = 0; k < M; k++)
                d[k] = __reduce_xor_sync(PAIR ? 0xFFFFu : FULL, p[k]);
        }
        if constexpr (PAIR)
            __syncwarp();
        if constexpr (W > 1) {
            uint32_t *sh = share + (N & 1) * W * 16;  // rewritten two barriers later
            uint32_t mine = 0;
#pragma unroll
            for (int k = 0; k < M; k++)
                mine = lane == k ? d[k] : mine;
            if (lane < M)
                sh[warp * 16 + lane] = mine;
            sync();
#pragma unroll
            for (int k = 0; k < M; k++)
                d[k] = 0;
#pragma unroll
            for (int w = 0; w < W; w++)
#pragma unroll
                for (int v = 0; v < (M + 3) / 4; v++) {
                    const uint4 x = reinterpret_cast<const uint4 *>(sh + w * 16)[v];
                    if (4 * v + 0 < M) d[4 * v + 0] ^= x.x;
                    if (4 * v + 1 < M) d[4 * v + 1] ^= x.y;
                    if (4 * v + 2 < M) d[4 * v + 2] ^= x.z;
                    if (4 * v + 3 < M) d[4 * v + 3] ^= x.w;
                }
        }
#pragma unroll
        for (int k = 0; k < M; k++)
            mne |= d[k];
        uint32_t ball[NQ];
        int Lmax = 0;
#pragma unroll
        for (int h = 0; h < NQ; h++) {
            const bool my_mle = ((mne >> (PAIR ? tid + 16 * h : lane)) & 1u) && (N >= 2 * Lq[h]);
            ball[h] = __ballot_sync(FULL, my_mle);
            Bd[h] = min(min(my_mle ? Lq[h] : Bd[h], T) + 1, T);
            Lq[h] = my_mle ? N + 1 - Lq[h] : Lq[h];
            Lmax = max(Lmax, Lq[h]);
        }
        // of a pair, each ballot has 16 bits of either tile
        const uint32_t mle = PAIR ? __byte_perm(ball[0], ball[NQ - 1], upper ? 0x7632 : 0x5410) : ball[0];
        const int Lb = min((int)__reduce_max_sync(FULL, (unsigned)Lmax), T);
        const int Bm = min(Bmax, T);
        uint32_t bs[H], ds[H];
        ksum<M>(bs, b);
        ksum<M>(ds, d);
        // After the step deg C <= L, so coefficients above the tile's new
        // largest L stay zero; B there only takes the swap (to C_i = 0) where
        // its degree bound reaches, and is zero above that.
        KAcc<M> acc;
        acc.clear();
        const int off = (R - (N % R)) % R;  // slot(i) = (i - N) mod R
        const int next = min(N + 1, 2 * T - 1);
        const int hi = max(Lb, Bm);
        const int srow = GLOBAL_SYN ? next % R : next;
#pragma unroll 1
        for (int i = first; (i & ~(PAIR ? 15 : 31)) <= hi; i += NT) {
            int slot = i + off;
            slot = slot >= R ? slot - R : slot;
            uint32_t *bp = ring + slot * SS;
            if (i <= Lb) {
                uint32_t *cp = cm + i * SS;
                const int sr = srow - i;
                const uint32_t *sp = syn + (GLOBAL_SYN && sr < 0 ? sr + R : sr) * SS;
                uint32_t bv[M], c[M], s[M], xs[H], ys[H], q[2 * M - 1];
#pragma unroll
                for (int k = 0; k < M; k++) {
                    bv[k] = bp[k];
                    c[k] = cp[k];
                    s[k] = sp[k];
                }
                KAcc<M> u;
                u.clear();
                ksum<M>(xs, c);
                u.mac(b, bs, c, xs);
                ksum<M>(xs, bv);
                u.mac(d, ds, bv, xs);
#pragma unroll
                for (int k = 0; k < M; k++)
                    bp[k] = (bv[k] & ~mle) | (c[k] & mle);
                u.combine(q);
                bs_reduce<M>(q);
#pragma unroll
                for (int k = 0; k < M; k++)
                    cp[k] = q[k];
                ksum<M>(xs, q);
                ksum<M>(ys, s);
                acc.mac(q, xs, s, ys);
            } else if (i <= Bm) {
#pragma unroll
                for (int k = 0; k < M; k++)
                    bp[k] &= ~mle;
            }
        }
#pragma unroll
        for (int k = 0; k < M; k++)
            b[k] = (b[k] & ~mle) | (d[k] & mle);
        const int freeslot = (R - ((N + 1) % R)) % R;
        if (tid < M)
            ring[freeslot * SS + tid] = 0;
        if (GLOBAL_SYN && tid < SS)  // over row N - t, which no later step reads
            syn[(N + 2) % R * SS + tid] = row;
        // (ciphertexts past the tile's count never take the swap: zero syndromes)
        unsigned Bm1 = 0;
#pragma unroll
        for (int h = 0; h < NQ; h++)
            Bm1 = max(Bm1, (PAIR ? tid + 16 * h : lane) < ntile ? (unsigned)Bd[h] : 0u);
        Bmax = (int)__reduce_max_sync(FULL, Bm1);
        acc.combine(p);
        bs_reduce<M>(p);
        if (W == 1)
            sync();  // W > 1: the next discrepancy's barrier
    }
    if (W > 1)
        sync();
}

}  // namespace cmd

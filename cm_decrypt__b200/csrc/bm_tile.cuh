// Berlekamp-Massey (bm.c:12-68) bitsliced across the 32 ciphertexts of a warp's
// tile: word bit q belongs to ciphertext q, lane l owns locator coefficients l,
// l + 32, ...  Coefficients, syndromes and B are rows of SS words in the warp's
// shared memory (SS = m made odd, so that lanes' rows meet no bank conflict; for
// m = 12 the 12-word rows of neighbouring lanes met four ways).
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

// One warp: syndromes syn -> locator coefficients C (both rows of SS words);
// ntile: ciphertexts of the tile (the others' syndromes are zero).
template <int S>
__device__ __forceinline__ void bm_tile_warp(const uint32_t *syn, uint32_t *ring, uint32_t *cm, int ntile, int lane)
{
    using Z = BmDims<S>;
    constexpr int M = Z::M, T = Z::T, SS = Z::SS, R = Z::R, H = KAcc<M>::H;
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    for (int v = lane; v < Z::C_WORDS; v += 32)
        cm[v] = v == 0 ? FULL : 0u;  // C = 1
    for (int v = lane; v < Z::RING_WORDS; v += 32)
        ring[v] = v == SS ? FULL : 0u;  // B = x
    uint32_t b[M], p[2 * M - 1];  // p: this lane's share of the discrepancy
#pragma unroll
    for (int k = 0; k < M; k++) {
        b[k] = k == 0 ? FULL : 0u;              // b = 1
        p[k] = lane == 0 ? syn[k] : 0u;         // d_0 = C_0 S_0
    }
    int Lq = 0;              // L of ciphertext `lane`
    int Bd = 1, Bmax = 1;    // bound on deg B of ciphertext `lane`; the tile's
    __syncwarp();
#pragma unroll 1
    for (int N = 0; N < 2 * T; N++) {
        uint32_t d[M], mne = 0;
#pragma unroll
        for (int k = 0; k < M; k++) {
            d[k] = __reduce_xor_sync(FULL, p[k]);
            mne |= d[k];
        }
        const bool my_mle = ((mne >> lane) & 1u) && (N >= 2 * Lq);
        const uint32_t mle = __ballot_sync(FULL, my_mle);
        const int Bdn = min(min(my_mle ? Lq : Bd, T) + 1, T);
        Lq = my_mle ? N + 1 - Lq : Lq;
        const int Lb = min((int)__reduce_max_sync(FULL, (unsigned)Lq), T);
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
#pragma unroll 1
        for (int i = lane; (i & ~31) <= hi; i += 32) {
            int slot = i + off;
            slot = slot >= R ? slot - R : slot;
            uint32_t *bp = ring + slot * SS;
            if (i <= Lb) {
                uint32_t *cp = cm + i * SS;
                const uint32_t *sp = syn + (next - i) * SS;
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
        if (lane < M)
            ring[freeslot * SS + lane] = 0;
        Bd = Bdn;
        // (lanes past the tile's count never take the swap: zero syndromes)
        Bmax = (int)__reduce_max_sync(FULL, lane < ntile ? (unsigned)Bd : 0u);
        acc.combine(p);
        bs_reduce<M>(p);
        __syncwarp();
    }
}

}  // namespace cmd

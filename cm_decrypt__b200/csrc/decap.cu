// KEM decapsulation around the decrypt path.  No counterpart in the
// reference, which encapsulates only: kem/common/core/operations.c:15-34
// computes C = [I | T] e and K = SHAKE256(1 || e || C) (32 bytes).  The
// Classic McEliece decapsulation inverts that with implicit rejection:
//
//   e = decrypt(C)                       (CMD_PATH_AUTO's kernels)
//   accept = padding bits mt..8*ct-1 of C are zero  &&  wt(e) == t
//            &&  C == [I | T] e          (e re-encodes to C)
//   K = SHAKE256(b || v || C),  b = accept,  v = accept ? e : s
//
// with T the systematic public key (derived once per key on the device from
// the key's support and Goppa polynomial by the key generation's elimination)
// and s the random string stored at the end of the secret key.
//
// k_reencode: the check, 64 ciphertexts a CTA, bitsliced across them.  T is the
// public key, so it may be used as an address; e is not, so it stays data:
//  1. the error rows are transposed, one word of 32 ciphertexts per column;
//  2. T's columns go five at a time: the CTA forms the 32 XOR combinations of
//     five error words in shared memory, and each row (a lane) adds the one its
//     five bits of T select.  The 32 combinations lie in 32 banks, so every
//     such read is one wavefront.  Bound by those reads (shared-memory pipe 71 %
//     busy): 288 us for 20,000 mceliece6688128 ciphertexts, against 766 us with
//     a lane a ciphertext and every column of T (52 words) masked by its bit;
//  3. row i must equal e_i + C_i; padding and weight checks.
// k_session_keys: SHAKE256 of the 1 + n/8 + ct byte preimage, one lane per
// ciphertext (Keccak-f[1600] as defined in FIPS 202; round constants and rotation
// offsets derived from the standard's definitions at compile time), the next
// block's words loaded during a permutation (110 us for the same batch; 175 us
// with the loads before each block); the preimage's v bytes are selected with
// masks.
// Every column of T and every word of e is read for every ciphertext, so the work
// and the addresses do not depend on e.
#include <cstring>
#include <mutex>

#include "engine.h"
#include "fused_impl.cuh"
#include "keccak.cuh"

namespace cmd {

namespace {

constexpr int DC_WARPS = 8;   // warps of a k_reencode block
constexpr int DC_CHUNK = 4;   // packed words of T per row and pass (24 groups of five columns)

template <int S> struct DecapDims {
    using P = Set<S>;
    static constexpr int MT = P::M * P::T;
    static constexpr int RG = (MT + 31) / 32;        // groups of 32 rows
    static constexpr int RP = 32 * RG;               // rows, padded
    static constexpr int XC = P::N - MT;             // columns of T
    static constexpr int NJ = (XC + 29) / 30;        // packed words a row: 30 columns each
    static constexpr int NCOL = MT + 30 * NJ;        // error words kept (zero past n)
    static constexpr int NB = P::N / 8;              // bytes of e and of s
    static constexpr int MSG = 1 + NB + P::CT;       // preimage bytes
    static constexpr int SMEM_WORDS = 2 * NCOL + 2 * DC_CHUNK * 6 * 32 * 2;
};

}  // namespace

struct DecapArgs {
    const uint8_t *cts;
    const uint32_t *err;       // error rows, nw words each
    uint16_t *weight;          // weights; k_reencode leaves 1 (accept) or 0 there
    const uint32_t *pkT;       // word j of row r of T at pkT[j * RP + r]: bit 5k + b = column 30j + 5k + b
    const uint8_t *s;          // the secret key's n/8-byte string s
    uint8_t *keys;             // 32 bytes per ciphertext
    uint8_t *accept;           // or null: 1 byte per ciphertext
    uint64_t count;
};

// 32 x 32 bit transpose across a warp (bit b of lane q's word to bit q of lane
// b's), five butterfly steps.
__device__ __forceinline__ uint32_t transpose32(uint32_t v, int lane)
{
    constexpr uint32_t M0[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int st = 0; st < 5; st++) {
        const int j = 16 >> st;
        const uint32_t y = __shfl_xor_sync(FULLMASK, v, j);
        const uint32_t keep = (lane & j) ? ~M0[st] : M0[st];
        const uint32_t t = (lane & j) ? (y >> j) : (y << j);
        v = (v & keep) | (t & ~keep);
    }
    return v;
}

// Bytes y, y + 1 (y even) of a ciphertext; its buffer may start at an odd address.
__device__ __forceinline__ uint32_t ct16(const uint8_t *ct, int y)
{
    return ((uintptr_t)ct & 1) == 0 ? *reinterpret_cast<const uint16_t *>(ct + y)
                                    : ct[y] | (uint32_t)ct[y + 1] << 8;
}

template <int S> __global__ void __launch_bounds__(DC_WARPS * 32, 3) k_reencode(DecapArgs a)
{
    using P = Set<S>;
    using Q = DecapDims<S>;
    constexpr int MT = Q::MT, NW = P::NW, RG = Q::RG, RP = Q::RP, NJ = Q::NJ, NCOL = Q::NCOL;
    constexpr int NR = (RG + DC_WARPS - 1) / DC_WARPS;  // row groups a warp
    constexpr int GW = DC_CHUNK * 6 * 32;               // combination words of a pass, per ciphertext word
    extern __shared__ __align__(16) uint32_t smem_dc[];
    __shared__ uint32_t s_bad[2];
    uint32_t *es = smem_dc, *comb = smem_dc + 2 * NCOL;  // es[h * NCOL + column], comb[pass & 1][h][group][32]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint64_t c0 = (uint64_t)blockIdx.x * 64;
    if (tid < 2)
        s_bad[tid] = 0;
    // ---- 1. error words ---------------------------------------------------------
    for (int v = warp; v < 2 * NW; v += DC_WARPS) {
        const int h = v >= NW, w = v - h * NW;
        const uint64_t c = c0 + 32 * h + lane;
        const uint32_t x = transpose32(c < a.count ? a.err[c * NW + w] : 0u, lane);
        if (32 * w + lane < NCOL)
            es[h * NCOL + 32 * w + lane] = x;
    }
    for (int v = 32 * NW + tid; v < NCOL; v += DC_WARPS * 32)
        es[v] = es[NCOL + v] = 0;
    __syncthreads();
    // ---- 2. T e -------------------------------------------------------------------
    uint32_t acc[NR][2];
#pragma unroll
    for (int i = 0; i < NR; i++)
        acc[i][0] = acc[i][1] = 0;
    const uint32_t *trow = a.pkT + 32 * warp + lane;  // row group i of this warp: + 32 * DC_WARPS * i
    auto form = [&](int j0) {  // the combinations of words j0 .. j0 + DC_CHUNK - 1
        uint32_t *dst = comb + (j0 / DC_CHUNK & 1) * 2 * GW;
        for (int v = warp; v < 2 * DC_CHUNK * 6; v += DC_WARPS) {
            const int h = v >= DC_CHUNK * 6, g = v - h * DC_CHUNK * 6, col = 30 * j0 + 5 * g;
            uint32_t x = 0;
            if (col < 30 * NJ) {
#pragma unroll
                for (int b = 0; b < 5; b++)
                    x = and_xor(x, es[h * NCOL + MT + col + b], 0u - ((uint32_t)lane >> b & 1u));
            }
            dst[h * GW + g * 32 + lane] = x;
        }
    };
    form(0);
    uint32_t t[NR];
#pragma unroll
    for (int i = 0; i < NR; i++)
        t[i] = warp + DC_WARPS * i < RG ? __ldg(trow + 32 * DC_WARPS * i) : 0u;
    __syncthreads();
#pragma unroll 1
    for (int j0 = 0; j0 < NJ; j0 += DC_CHUNK) {
        if (j0 + DC_CHUNK < NJ)
            form(j0 + DC_CHUNK);
        const uint8_t *cb = reinterpret_cast<const uint8_t *>(comb + (j0 / DC_CHUNK & 1) * 2 * GW);
#pragma unroll 1
        for (int j = j0; j < j0 + DC_CHUNK && j < NJ; j++, cb += 6 * 32 * 4) {
            uint32_t nx[NR];
#pragma unroll
            for (int i = 0; i < NR; i++)
                nx[i] = j + 1 < NJ && warp + DC_WARPS * i < RG ? __ldg(trow + (size_t)(j + 1) * RP + 32 * DC_WARPS * i)
                                                               : 0u;
#pragma unroll
            for (int k = 0; k < 6; k++)
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const uint32_t o = (k == 0 ? t[i] << 2 : t[i] >> (5 * k - 2)) & 0x7Cu;
                    acc[i][0] ^= *reinterpret_cast<const uint32_t *>(cb + k * 128 + o);
                    acc[i][1] ^= *reinterpret_cast<const uint32_t *>(cb + k * 128 + GW * 4 + o);
                }
#pragma unroll
            for (int i = 0; i < NR; i++)
                t[i] = nx[i];
        }
        __syncthreads();
    }
    // ---- 3. acceptance ----------------------------------------------------------
    uint32_t bad[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < NR; i++) {
        const int rg = warp + DC_WARPS * i, r = 32 * rg + lane;
        if (rg >= RG)
            break;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint64_t c = c0 + 32 * h + lane;
            uint32_t x = 0;
            if (c < a.count) {
                const uint8_t *ct = a.cts + c * P::CT;
                x = ct16(ct, 4 * rg);
                if (4 * rg + 2 < P::CT)
                    x |= ct16(ct, 4 * rg + 2) << 16;
            }
            x = transpose32(x, lane);  // row r of C; rows mt.. are padding, which must be zero
            bad[h] |= r < MT ? x ^ es[h * NCOL + r] ^ acc[i][h] : r < 8 * P::CT ? x : 0u;
        }
    }
    bad[0] = __reduce_or_sync(FULLMASK, bad[0]);
    bad[1] = __reduce_or_sync(FULLMASK, bad[1]);
    if (lane == 0) {
        atomicOr(&s_bad[0], bad[0]);
        atomicOr(&s_bad[1], bad[1]);
    }
    __syncthreads();
    const uint64_t c = c0 + tid;
    if (tid < 64 && c < a.count) {
        const bool ok = (s_bad[tid >> 5] >> lane & 1u) == 0 && a.weight[c] == P::T;
        a.weight[c] = ok ? 1 : 0;
        if (a.accept)
            a.accept[c] = ok ? 1 : 0;
    }
}

constexpr int KEY_THREADS = 64;  // small blocks: a batch spreads over the SMs evenly

template <int S> __global__ void __launch_bounds__(KEY_THREADS) k_session_keys(DecapArgs a)
{
    using P = Set<S>;
    using Q = DecapDims<S>;
    const uint64_t cc = (uint64_t)blockIdx.x * KEY_THREADS + threadIdx.x;
    if (cc >= a.count)
        return;
    const uint32_t *erow = a.err + cc * P::NW;
    const uint8_t *ct = a.cts + cc * P::CT;
    const uint32_t okm = 0u - (uint32_t)a.weight[cc];
    // K = SHAKE256(b || v || C), 32 bytes.
    // preimage byte 0: b; then v, C and the pad10*1 padding with the SHAKE domain
    // bits (0x1F ... 0x80) over whole 136-byte blocks.  The stream after byte 0 is
    // read in words (v selected by mask from e and s) and shifted by that byte:
    // byte by byte, this step took most of the kernel.
    constexpr int RATE = 136, NB = Q::NB, END = NB + P::CT;
    constexpr int NBLK = Q::MSG / RATE + 1;
    static_assert(NB % 2 == 0 && P::CT % 2 == 0, "16-bit units");
    const uint16_t *s16 = reinterpret_cast<const uint16_t *>(a.s);  // an even offset of the aligned secret key
    auto half = [&](int x) -> uint32_t {  // bytes x, x + 1 (x even) of v || C || padding
        if (x < NB)
            return ((erow[x >> 2] >> (8 * (x & 2)) & okm) | (s16[x >> 1] & ~okm)) & 0xFFFFu;
        if (x < END)
            return ct16(ct, x - NB);
        return x == END ? 0x1Fu : 0u;
    };
    auto word = [&](int x) -> uint32_t {  // bytes x .. x + 3 (x a multiple of 4)
        if (x + 4 <= NB)
            return (erow[x >> 2] & okm) | ((s16[x >> 1] | (uint32_t)s16[(x >> 1) + 1] << 16) & ~okm);
        return half(x) | half(x + 2) << 16;
    };
    uint64_t A[25];
#pragma unroll
    for (int i = 0; i < 25; i++)
        A[i] = 0;
    uint32_t prev = okm & 0x01000000u;  // byte 0, as the last byte of a word before the stream
    // the next block's words, on their way during a permutation; blocks inside v
    // without a branch a word, so that their loads go out together
    uint32_t nx[RATE / 4];
    auto fetch = [&](int blk) {
        if ((blk + 1) * RATE <= NB) {
#pragma unroll
            for (int l = 0; l < RATE / 4; l++) {
                const int w = blk * (RATE / 4) + l;
                nx[l] = (erow[w] & okm) | ((s16[2 * w] | (uint32_t)s16[2 * w + 1] << 16) & ~okm);
            }
        } else {
#pragma unroll
            for (int l = 0; l < RATE / 4; l++)
                nx[l] = word(blk * RATE + 4 * l);
        }
    };
    fetch(0);
#pragma unroll 1
    for (int blk = 0; blk < NBLK; blk++) {
#pragma unroll
        for (int l = 0; l < RATE / 8; l++) {  // static lane index: A stays in registers
            const uint32_t w0 = nx[2 * l], w1 = nx[2 * l + 1];
            const uint32_t lo = __funnelshift_l(prev, w0, 8);
            uint32_t hi = __funnelshift_l(w0, w1, 8);
            if (l == RATE / 8 - 1 && blk == NBLK - 1)
                hi |= 0x80000000u;
            A[l] ^= (uint64_t)hi << 32 | lo;
            prev = w1;
        }
        if (blk + 1 < NBLK)
            fetch(blk + 1);
        keccak_f(A);
    }
    uint64_t *out = reinterpret_cast<uint64_t *>(a.keys + cc * 32);
#pragma unroll
    for (int i = 0; i < 4; i++)
        out[i] = A[i];
}

size_t decap_pk_words(int set)
{
    return dispatch_set(set, [&]<int S>() -> size_t { return (size_t)DecapDims<S>::NJ * DecapDims<S>::RP; });
}

cudaError_t launch_decap(int set, const uint8_t *d_cts, const uint32_t *d_err, uint16_t *d_w, const uint32_t *d_pk,
                         const uint8_t *d_s, uint8_t *d_keys, uint8_t *d_accept, size_t count, cudaStream_t s,
                         LaunchCounter lc)
{
    if (count == 0)
        return cudaSuccess;
    DecapArgs a{d_cts, d_err, d_w, d_pk, d_s, d_keys, d_accept, count};
    return dispatch_set(set, [&]<int S>() -> cudaError_t {
        constexpr int smem = 4 * DecapDims<S>::SMEM_WORDS;
        static bool given[64] = {};  // per device
        int dev = 0;
        cudaGetDevice(&dev);
        if (!given[dev & 63]) {
            const cudaError_t e =
                cudaFuncSetAttribute(k_reencode<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess)
                return e;
            given[dev & 63] = true;
        }
        k_reencode<S><<<(unsigned)((count + 63) / 64), DC_WARPS * 32, smem, s>>>(a);
        k_session_keys<S><<<(unsigned)((count + KEY_THREADS - 1) / KEY_THREADS), KEY_THREADS, 0, s>>>(a);
        lc.bump(2);
        return cudaGetLastError();
    });
}

// A device batch; the key is prepared.  Caller holds eng->mu.
static int run_decap(cmd_engine *eng, cmd_key *key, const uint8_t *d_cts, size_t count, uint8_t *d_keys,
                     uint8_t *d_accept, cudaStream_t s)
{
    const SetInfo si = set_info(key->dev.set);
    const size_t words = count * si.nw;
    int rc = eng->scratch.begin(eng, words * 4 + count * 2 + 256, s);
    if (rc)
        return rc;
    uint32_t *d_err = static_cast<uint32_t *>(eng->scratch.ptr);
    uint16_t *d_w = reinterpret_cast<uint16_t *>(d_err + words);
    cudaError_t e = cudaSuccess;
    if ((rc = run_device(eng, key, CMD_PATH_AUTO, d_cts, count, d_err, d_w, s)) == CMD_OK) {
        const uint8_t *d_s = key->dev.sk + 40 + 2 * si.t + si.cond;
        e = launch_decap(key->dev.set, d_cts, d_err, d_w, key->pk, d_s, d_keys, d_accept, count, s,
                         LaunchCounter{&eng->launches});
    }
    const int r = eng->scratch.end(s, e);  // the rows are read up to here
    return rc ? rc : r;
}

}  // namespace cmd

using namespace cmd;

extern "C" {

int cmd_key_prepare_decap(cmd_engine *eng, cmd_key *key)
{
    if (!eng || !key || key->eng != eng)
        return CMD_E_ARG;
    // one preparation at a time per key, so that two first calls for a key
    // derive its columns once (keys of other engines and devices prepare in
    // parallel); taken before eng->mu, which kg_pubkey_rows takes
    std::lock_guard<std::mutex> lk(key->prep_mu);
    if (key->pk)
        return CMD_OK;
    const int set = key->dev.set;
    const size_t bytes = decap_pk_words(set) * 4;
    const int rp = dispatch_set(set, [&]<int S>() { return DecapDims<S>::RP; });
    void *p = nullptr;
    int rc = device_alloc(eng, &p, bytes, "public key columns", "public key does not fit the engine HBM budget");
    if (rc)
        return rc;
    // the key's parity-check matrix from its device support and Goppa
    // polynomial, reduced on the device
    rc = kg_pubkey_rows(eng, set, key->dev.L, key->dev.g, static_cast<uint32_t *>(p), rp);
    if (rc) {
        cudaFree(p);
        budget_give(eng, bytes);
        return rc;
    }
    key->pk = static_cast<uint32_t *>(p);
    key->pk_bytes = bytes;
    return CMD_OK;
}

int cmd_kem_decap_device(cmd_engine *eng, cmd_key *key, const uint8_t *d_cts, size_t count, uint8_t *d_keys,
                         uint8_t *d_accept, void *stream)
{
    if (!eng || !key || key->eng != eng || (count && (!d_cts || !d_keys)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    int rc = cmd_key_prepare_decap(eng, key);
    if (rc)
        return rc;
    cudaSetDevice(eng->device);
    std::lock_guard<std::mutex> lk(eng->mu);
    return run_decap(eng, key, d_cts, count, d_keys, d_accept, stream ? (cudaStream_t)stream : eng->stream);
}

int cmd_kem_decap(cmd_engine *eng, cmd_key *key, const uint8_t *h_cts, size_t count, uint8_t *h_keys,
                  uint8_t *h_accept)
{
    if (!eng || !key || key->eng != eng || (count && (!h_cts || !h_keys)))
        return CMD_E_ARG;
    if (count == 0)
        return CMD_OK;
    int rc = cmd_key_prepare_decap(eng, key);
    if (rc)
        return rc;
    const SetInfo si = set_info(key->dev.set);
    cudaSetDevice(eng->device);
    const size_t chunk = std::min<size_t>(count, (size_t)1 << 20);
    std::lock_guard<std::mutex> lk(eng->mu);  // up to the last copy: calls share the buffers below
    if ((rc = eng->io.reserve(eng, chunk * (si.ct + 32 + 1) + 1024)))
        return rc;
    uint8_t *d_cts = static_cast<uint8_t *>(eng->io.ptr), *d_keys = d_cts + (chunk * si.ct + 255) / 256 * 256,
            *d_acc = d_keys + chunk * 32;
    cudaStream_t s = eng->stream;
    for (size_t c0 = 0; c0 < count; c0 += chunk) {
        const size_t n = std::min(chunk, count - c0);
        cudaError_t e = cudaMemcpyAsync(d_cts, h_cts + c0 * si.ct, n * si.ct, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMemcpyAsync(cts H2D)");
        if ((rc = run_decap(eng, key, d_cts, n, d_keys, d_acc, s)))
            return rc;
        e = cudaMemcpyAsync(h_keys + c0 * 32, d_keys, n * 32, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && h_accept)
            e = cudaMemcpyAsync(h_accept + c0, d_acc, n, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(s);
        if (e != cudaSuccess)
            return cuda_fail(e, "decapsulation D2H");
    }
    return CMD_OK;
}

}  // extern "C"

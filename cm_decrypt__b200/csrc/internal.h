// Engine-internal declarations shared by the CUDA launchers and the C ABI.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <string>

#include "cmd_b200.h"
#include "params.h"

namespace cmd {

// Device-resident expanded key: one allocation carved into these arrays.
struct KeyDev {
    int set = 0;
    uint16_t *L = nullptr;      // support, n entries (support_gen output)
    uint16_t *g = nullptr;      // Goppa polynomial, t+1 coefficients, g[t] = 1
    uint16_t *ginv2 = nullptr;  // 1/g(L_i)^2 for i < n (0 where g(L_i) = 0)
    uint32_t *tab = nullptr;    // syndrome table, sb rows of twp (t rounded up to
                                // 4) words; word w < t of row b packs
                                // L_b^{2w}/g^2 (low) and L_b^{2w+1}/g^2 (high):
                                // util.c:86-100 values, rows 16-byte aligned
    uint32_t *tabd = nullptr;   // the same table, dense: sb rows of twd words,
                                // bit j*m + k of row b = bit k of L_b^j/g^2
                                // (the fused kernel's syndrome source)
    uint32_t *Lbs = nullptr;    // bitsliced support, plane-major [m][nw]:
                                // bit p of Lbs[k*nw+w] = bit k of L[32w+p]
    uint32_t *bctl = nullptr;   // Benes network as swap masks, [2m-1][2^(m-5)]:
                                // bit b of bctl[l*2^(m-5)+w] set when layer l
                                // exchanges position 32w+b (the pair's lower
                                // element) with its partner
    uint32_t *wfft = nullptr;   // 1/g(a)^2 at every field element a in the
                                // additive FFT's position order, bitsliced
                                // plane-major [m][2^(m-5)]: bit b of word w is
                                // the element a = bitrev_m(32w + b)
    uint8_t *sk = nullptr;      // device copy of the secret key bytes
};

// Records a launch against an engine counter (count of our kernels).
struct LaunchCounter {
    std::atomic<uint64_t> *ctr;
    void bump(uint64_t n = 1) const
    {
        if (ctr)
            ctr->fetch_add(n, std::memory_order_relaxed);
    }
};

cudaError_t launch_key_expand(const KeyDev &k, cudaStream_t s, LaunchCounter lc);
// Words of KeyDev::bctl for one set.
inline size_t benes_mask_words(const SetInfo &si) { return (size_t)(2 * si.m - 1) << (si.m - 5); }
// Words of KeyDev::wfft for one set.
inline size_t fft_weight_words(const SetInfo &si) { return (size_t)si.m << (si.m - 5); }

cudaError_t launch_synd_plain(const KeyDev &k, const uint8_t *d_cts, size_t count,
                              uint32_t *d_synd, cudaStream_t s, LaunchCounter lc);
cudaError_t launch_bm_plain(int set, const uint16_t *d_synd, size_t count, uint16_t *d_loc,
                            cudaStream_t s, LaunchCounter lc);
cudaError_t launch_root_plain(const KeyDev &k, const uint16_t *d_loc, size_t count,
                              uint32_t *d_err, uint16_t *d_weight, cudaStream_t s,
                              LaunchCounter lc, int num_sms);
cudaError_t launch_root_images(const KeyDev &k, const uint16_t *d_loc, size_t count,
                               uint16_t *d_images, cudaStream_t s, LaunchCounter lc);
cudaError_t preload_plain_kernels();

// Fused path: one work item = up to 32 ciphertexts of one key.
struct FusedTile {
    uint32_t key;     // index into the key table
    uint32_t count;   // 1..32
    uint64_t first;   // index of the first ciphertext of the tile in the
                      // ciphertext index list (mixed) or the batch (single)
};
struct FusedKeyRef {
    int32_t set;
    int32_t pad;
    const uint32_t *tab;
    const uint32_t *Lbs;
    const uint32_t *bctl;
};

// Additive-FFT evaluation plan of one parameter set (fft_plan.cpp): constant
// tables shared by every key of the set.
//   scalpow[d*256 + i]: b_d^i, the radix-conversion scale of depth d;
//   tw[k*2^(m-5) + off_d + u]: plane k of twiddle word u of depth d (off_d =
//   the sum of the word counts 2^(m-e-6) of the depths e < d); planes m, m + 1,
//   ... are the half sums plane k ^ plane k + (m+1)/2.
struct FftPlanDev {
    const uint16_t *scalpow;
    const uint32_t *tw;
};
struct FusedArgs {
    const FusedTile *tiles;        // device list of rounds; null = implicit
                                   // rounds over one key: round r covers
                                   // ciphertexts [r*round_cts, +round_cts)
    uint32_t ntiles;               // number of rounds
    uint32_t round_cts;            // implicit mode: ciphertexts per round
    uint64_t total;                // implicit mode: batch size
    const FusedKeyRef *keys;       // device key table (null in implicit mode)
    FusedKeyRef key0;              // implicit mode: the one key
    const uint8_t *cts;            // ciphertext base pointer
    const uint64_t *ct_off;        // per-ciphertext byte offsets, or null
    const uint64_t *err_off;       // per-ciphertext error-row word offsets, or null
    const uint32_t *order;         // ciphertext index per round slot, or null
    uint32_t *err;
    uint16_t *weight;
    uint32_t *tile_counter;        // zeroed before the launch
    int single_set;                // >= 0: every round has this set
    uint32_t err_stride;           // words per error row when err_off is null
    uint16_t *pos;                 // or null: per ciphertext t+1 u16, the weight
                                   // then the error positions ascending, 0xFFFF after
    uint32_t pos_stride;           // u16 per positions row
    uint8_t *err_packed;           // or null: error rows of n/8 bytes back to back
                                   // (a host-mapped buffer), row c at c * n/8
    FftPlanDev fft[NSETS];         // root-search plans, indexed by set
};
cudaError_t launch_fused(const FusedArgs &a, int grid, int warps_per_block, cudaStream_t s,
                         LaunchCounter lc);

// One key's batch in four kernels (staged.cu): error rows at the set's nw stride,
// weights, positions rows (FusedArgs::pos), each or null.  d_scratch:
// staged_scratch_words(set, count) words.  many_parts: one of more than two parts of
// a batch, on several streams.
cudaError_t launch_staged(const KeyDev &k, const uint8_t *d_cts, uint32_t count, uint32_t *d_scratch, uint32_t *d_err,
                          uint16_t *d_weight, uint16_t *d_pos, const FftPlanDev &plan, int num_sms, bool many_parts,
                          cudaStream_t s, LaunchCounter lc);
size_t staged_scratch_words(int set, size_t count);
// The same for the ciphertexts of one set in a mixed batch: `blocks` and `tiles`
// cut the slots of `order` (a key's slots contiguous) into syndrome blocks of up
// to staged_block_tiles tiles and tiles of up to 32 slots, each of one key.
struct StagedPiece {
    uint32_t key;    // index into keys
    uint32_t count;  // slots
    uint32_t first;  // first slot
    uint32_t tile0;  // blocks: their first tile
};
struct StagedMixed {
    const StagedPiece *blocks = nullptr, *tiles = nullptr;
    const FusedKeyRef *keys = nullptr;
    const uint32_t *order = nullptr;    // ciphertext index of a slot
    const uint64_t *ct_off = nullptr;   // by ciphertext: bytes
    const uint64_t *err_off = nullptr;  // words
};
constexpr uint32_t staged_block_tiles = 8;
cudaError_t launch_staged_mixed(int set, const StagedMixed &mx, uint32_t nblocks, uint32_t ntiles,
                                const uint8_t *d_cts, uint32_t *d_scratch, uint32_t *d_err, uint16_t *d_weight,
                                const FftPlanDev &plan, int num_sms, cudaStream_t s, LaunchCounter lc);

// Latency path (serving loop; latency.cu): one work item per ciphertext.
struct LatItem {
    const uint32_t *wfft; // key's syndrome weights in FFT order (KeyDev::wfft)
    const uint32_t *bctl; // key's support-network swap masks
    uint32_t ct_off;      // byte offset of the ciphertext in the batch
    uint32_t err_off;     // word offset of the error row in the batch
    int32_t set;
    int32_t pad;
    uint8_t *row;         // or the packed n/8-byte error row, stored here (GPU-mapped host memory)
};
// Tile path: ntiles tiles of 32 item slots (LatItem.pad = tile count, padding
// slots set -1).  d_scratch holds ntiles * TILE_SCRATCH_WORDS words: each
// tile's radix-converted locators (bitsliced, 16 words per entry), then the
// transposed-FFT sums of its ciphertexts (2^D' u16 entries x 32 slots).
constexpr int TILE_LOC_WORDS = 256 * 16;
constexpr int TILE_SUM_WORDS = 256 * 32 / 2;
constexpr int TILE_SCRATCH_WORDS = TILE_LOC_WORDS + TILE_SUM_WORDS;
struct FftPlans {
    FftPlanDev p[NSETS];
};
// live: ciphertexts among the slots; beside: those of batches in flight on other
// streams.  Small batches take the per-ciphertext kernels below, while what is in
// flight stays within CT_IN_FLIGHT_PER_SM an SM: they finish sooner on a GPU with room,
// but do more work for a ciphertext than the tile kernels.  Without that bound the
// server, 1,024 keys, kept a queue once it had one: at 8 M requests/s p50 1.4 instead
// of 0.42 ms in some runs, at 9 M 2.2 ms in all.  At 36 an SM p50 / p99 0.42 / 0.55 at
// 8 M (0.77 / 1.0), 0.46 / 0.60 at 8.5 M (0.79 / 1.03), 0.76 / 1.01 at 9 M (0.83 /
// 1.07), 0.80 / 1.05 at 9.5 M (0.88 / 1.11), 0.84 / 1.09 at 10 M (0.95 / 1.17), in
// brackets the tile kernels alone; 24 lets 7 M go to them (0.69 against 0.37), 44
// raises p99 at 9 M to 1.17 ms.
cudaError_t launch_tile_path(const void *d_items, const uint8_t *d_cts, uint32_t ntiles, uint32_t live,
                             uint32_t beside, uint32_t *d_scratch, uint32_t *d_err, uint16_t *d_weight,
                             const FftPlans &plans, int num_sms, cudaStream_t s, LaunchCounter lc);
// The tile path over one key's batch (ciphertexts at the set's ct stride,
// error rows at its nw stride); with d_synd, only the syndromes (rows of 2t
// u16).  d_scratch: tile_single_scratch_words(count) words.  d_pos (positions
// rows): only for batches of up to CT_PER_SM an SM.
cudaError_t launch_tile_single(const KeyDev &k, const uint8_t *d_cts, size_t count, uint32_t *d_scratch,
                               uint32_t *d_err, uint16_t *d_weight, uint16_t *d_pos, uint16_t *d_synd,
                               const FftPlans &plans, int num_sms, cudaStream_t s, LaunchCounter lc);
size_t tile_single_scratch_words(size_t count);
// The per-ciphertext kernels (single.cu).  Up to CT_ONE_LAUNCH live
// ciphertexts run in one launch; more, up to CT_PER_SM an SM, in three with
// d_mid (256 u16 per slot) between them.  launch_ct_items: nslots items (set
// -1: skipped), `live` of them in use.  launch_ct_one: count <= CT_ONE_LAUNCH
// ciphertexts of one key at the set's strides.  d_pos: rows of t+1 u16 by slot
// (FusedArgs::pos), of one set.
constexpr uint32_t CT_ONE_LAUNCH = 64, CT_PER_SM = 24, CT_IN_FLIGHT_PER_SM = 36;
cudaError_t launch_ct_items(const LatItem *d_items, const uint8_t *d_cts, uint32_t nslots, uint32_t live,
                            uint16_t *d_mid, uint32_t *d_err, uint16_t *d_weight, uint16_t *d_pos,
                            const FftPlans &plans, int num_sms, cudaStream_t s, LaunchCounter lc);
cudaError_t launch_ct_one(const KeyDev &k, const uint8_t *d_cts, uint32_t count, uint32_t *d_err, uint16_t *d_weight,
                          uint16_t *d_pos, const FftPlans &plans, cudaStream_t s, LaunchCounter lc);

void set_last_error(const std::string &msg);

}  // namespace cmd

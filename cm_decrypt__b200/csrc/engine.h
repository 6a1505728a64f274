// Engine and key objects behind the opaque C handles, plus the helpers the
// batch, tuning and serving code share.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "internal.h"

struct cmd_engine;

namespace cmd {

// Growable device buffer charged against the engine's HBM budget.
struct Scratch {
    void *ptr = nullptr;
    size_t cap = 0;
    cudaEvent_t done = nullptr;  // after the last use between begin and end
    bool captured = false;       // in a graph: growing leaves this block to the engine
    // no_memory: returned when the budget allows the growth but the device's memory
    // does not (others use it, too); CMD_E_BUDGET from callers that can do without.
    int reserve(cmd_engine *eng, size_t bytes, int no_memory = CMD_E_CUDA);
    // Around work on a caller's stream that uses the buffer: reserves it and orders
    // s after its last use on any stream; marks this use (also after an error e).
    // A stream under capture neither waits nor marks; its graph keeps the address, so
    // the block stays until the engine goes.
    int begin(cmd_engine *eng, size_t bytes, cudaStream_t s, int no_memory = CMD_E_CUDA);
    int end(cudaStream_t s, cudaError_t e = cudaSuccess);
    void release(cmd_engine *eng);
};

// Growable pinned host buffer (staging for host-pointer calls).
struct HostScratch {
    void *ptr = nullptr;
    size_t cap = 0;
    int reserve(size_t bytes);
    void release();
};

// Fused-kernel launch configuration chosen per parameter set.
struct FusedConfig {
    int wpb = 8;          // warps per CTA (4 or 8)
    bool balanced = true; // equal-share rounds (see round_size in batch.cu)
    bool tuned = false;
    double ns_per_ct = 0; // measured by the tuner
    uint32_t tile_below = 0;  // CMD_PATH_AUTO: batches smaller than this take
                              // the small-batch kernels (launch_tile_single)
                              // instead of the staged ones; batches within
                              // the per-ciphertext kernels' reach take them
                              // at any value (takes_small in engine.cu)
};

int cuda_fail(cudaError_t e, const char *what);
// T of the public key [I | T] of a key, from its device support d_L (n entries) and
// Goppa polynomial d_g (t + 1 coefficients): bit i of d_rows[j * rp + r] is column
// 30 j + i of row r, rp >= mt.  CMD_E_ARG when the key's parity-check matrix has no
// systematic form.  Takes eng->mu.
int kg_pubkey_rows(cmd_engine *eng, int set, const uint16_t *d_L, const uint16_t *d_g, uint32_t *d_rows, int rp);
bool valid_set(int set);
bool budget_take(cmd_engine *eng, size_t bytes);
// The same for what the engine holds longer than a call, which the scratch kept for
// CMD_PATH_AUTO makes room for when it has to (the calls that it serves can do
// without); and device memory so charged: CMD_E_BUDGET with the message `over`, or
// CMD_E_CUDA.  Not with eng->mu held.
bool budget_take_first(cmd_engine *eng, size_t bytes);
int device_alloc(cmd_engine *eng, void **p, size_t bytes, const char *what, const char *over);
// Device address of GPU-mapped host memory [h, h + bytes) (2-byte aligned,
// one contiguous mapping), or null.
uint8_t *device_view(uint8_t *h, size_t bytes);
void budget_give(cmd_engine *eng, size_t bytes);

// d_pos: with CMD_PATH_AUTO only, positions rows instead of error rows.
int run_device(cmd_engine *eng, const cmd_key *key, cmd_path path, const uint8_t *d_cts, size_t count,
               uint32_t *d_err, uint16_t *d_weight, cudaStream_t s, uint16_t *d_pos = nullptr);
int run_fused_single(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                     uint16_t *d_weight, cudaStream_t s, uint16_t *d_pos = nullptr);
// The staged kernels over one key's device batch (see engine.cu): err/weight or
// pos, each or null.  CMD_E_BUDGET when their scratch does not fit the budget or
// the device.
int run_staged(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
               uint16_t *d_weight, uint16_t *d_pos, cudaStream_t s);
// Around staged launches on s (ns = 1) or on the first ns piece streams: reserves
// the scratch, orders it after its last use on another stream, forks; joins (also
// after an error e) and marks the scratch's use.
int staged_begin(cmd_engine *eng, size_t bytes, int ns, cudaStream_t s);
int staged_end(cmd_engine *eng, int ns, cudaStream_t s, cudaError_t e);
// Explicit work counter and round schedule (balanced: -1 = the tuned choice,
// 0 = full rounds, 1 = equal shares; round_cts > 0 overrides all three with
// rounds of that many ciphertexts, a multiple of 32 from fused_round).
// err_packed: or null, a device-writable view of rows of n/8 bytes back to
// back (a host-mapped buffer the kernel fills directly).
int run_fused_counter(cmd_engine *eng, const cmd_key *key, const uint8_t *d_cts, size_t count, uint32_t *d_err,
                      uint16_t *d_weight, cudaStream_t s, uint32_t *counter, uint16_t *d_pos, int balanced,
                      uint32_t round_cts = 0, uint8_t *err_packed = nullptr);
// Ciphertexts per round of one launch over `count` ciphertexts of `set` under
// the tuned schedule.
uint32_t fused_round(cmd_engine *eng, int set, size_t count);
constexpr int BATCH_STREAMS = 8;      // pieces of a host-buffer batch in flight
// cmd_engine::tile_counter: one u32 for calls that wait for their launches, one a
// piece of theirs, then a ring for launches on callers' streams.
constexpr int COUNTER_RING = 16, COUNTER_RING0 = 1 + BATCH_STREAMS, TILE_COUNTERS = COUNTER_RING0 + COUNTER_RING;
bool capturing(cudaStream_t s);
// While it lives, calls of this thread that take no part in a capture (allocations, work
// on other streams) may be made beside one.
struct BesideCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
// Device memory for a graph, kept until the engine goes: CMD_E_BUDGET, CMD_E_CUDA.  Beside
// a capture; with eng->mu held.
int graph_alloc(cmd_engine *eng, size_t bytes, void **p);
// Around a fused launch on a caller's stream: a work counter that no other launch in
// flight uses, the next of the ring once its last launch has ended.  Under capture
// the counter stays the captured launch's own, since a graph may be replayed at
// any time.
struct TileCounter {
    uint32_t *ptr = nullptr;
    cudaEvent_t done = nullptr;  // null under capture
    int begin(cmd_engine *eng, cudaStream_t s);
    int end(cudaStream_t s, int rc);  // also after an error rc
};
constexpr int STAGED_STREAMS = 4;     // parts of a staged device batch in flight
int ensure_piece_streams(cmd_engine *eng);
size_t fused_smem(int set, int wpb);
size_t smem_limit_bytes();
int fused_blocks_per_sm(int single_set, int wpb, size_t smem);
int fused_grid(cmd_engine *eng, int single_set, int wpb, size_t smem, uint64_t rounds);
int mixed_single_set(const int *key_set, const uint32_t *key_idx, size_t count);
void plan_mixed(const int *key_set, size_t nkeys, const uint32_t *key_idx, size_t count, uint32_t R,
                std::vector<uint32_t> &order, std::vector<FusedTile> &tiles);
// Root-search tables (fft_plan.cpp): uploaded once per engine, budget-charged.
int upload_fft_plans(cmd_engine *eng);
// No-allocation path (noalloc.cu): with `device` current, looks up the
// scratch array's device address and loads the plain kernels, so that
// cmd_decrypt_plain_noalloc itself loads and allocates nothing.
int noalloc_setup(int device);
void release_fft_plans(cmd_engine *eng);
inline FusedKeyRef key_ref(const KeyDev &k) { return FusedKeyRef{k.set, 0, k.tabd, k.Lbs, k.bctl}; }

}  // namespace cmd

struct cmd_engine {
    int device = 0;
    int num_sms = 0;
    char gpu_name[256] = {0};
    size_t budget = 0;
    std::atomic<size_t> used{0};
    cudaStream_t stream = nullptr;
    std::mutex mu;                 // serialises calls that share scratch
    cmd::Scratch scratch;          // intermediates of the plain and tile paths, a decapsulation's error rows
    cmd::Scratch io;               // device staging for host-buffer calls
    cmd::Scratch fused;            // fused-kernel work lists
    cmd::Scratch staged;           // staged kernels' intermediates, one part per piece stream,
                                   // and CMD_PATH_AUTO's small batches'
    cudaEvent_t staged_fork = nullptr, staged_join[cmd::STAGED_STREAMS] = {};  // created on first use
    cmd::Scratch keygen;           // key-generation workspace (kept between calls)
    std::vector<void *> graph_blocks;  // outgrown scratch and work lists that graphs may use
    size_t graph_block_bytes = 0;
    cmd::HostScratch host_scratch; // pinned staging
    uint32_t *tile_counter = nullptr;  // the fused kernel's work counters
    cudaEvent_t counter_done[cmd::COUNTER_RING] = {};  // created on first use
    unsigned counter_next = 0;
    std::vector<uint32_t *> graph_counters;  // blocks of counters of captured launches
    unsigned graph_counters_left = 0;        // in the last block
    cudaStream_t piece_stream[cmd::BATCH_STREAMS] = {};  // host-buffer batches, created on first use
    std::atomic<uint64_t> launches{0};
    cmd::FusedConfig fcfg[cmd::NSETS];
    cmd::FusedConfig fcfg_mixed;
    cmd::FftPlanDev fft[cmd::NSETS] = {};  // per-set root-search tables
    void *fft_mem = nullptr;
    size_t fft_bytes = 0;
};

namespace cmd {
inline void fill_fft(FusedArgs &a, const cmd_engine *eng)
{
    for (int s = 0; s < NSETS; s++)
        a.fft[s] = eng->fft[s];
}
}  // namespace cmd

struct cmd_key {
    cmd_engine *eng = nullptr;
    cmd::KeyDev dev;
    void *block = nullptr;
    size_t bytes = 0;
    uint32_t *pk = nullptr;  // decapsulation: T block of the public key (kg_pubkey_rows)
    size_t pk_bytes = 0;
    std::mutex prep_mu;      // cmd_key_prepare_decap, per key (before eng->mu)
};

// A CUDA runtime for host tests: device memory is host memory, kernels do not run,
// and every operation is recorded with a vector clock, so that a test can ask
// whether one operation is ordered before another whatever the streams' timing.
// Allocations can be made to fail, and stream capture refuses what CUDA refuses.
// Linked with the engine's own objects in place of the CUDA runtime library.
#include <cuda_runtime_api.h>
#include <unistd.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

namespace {

using Clock = std::map<int, uint64_t>;  // operations seen of each stream

void join(Clock &to, const Clock &from)
{
    for (const auto &[s, n] : from)
        if (to[s] < n)
            to[s] = n;
}

struct Event {
    Clock at;
    int capture = 0;  // the capture it was last recorded in
};
struct Stream {
    int id = 0;
    Clock seen;
    int capture = 0;  // id of the capture in progress
    bool global = false, broken = false;
};
struct Op {
    int call, stream;
    uint64_t index;  // on its stream, from 1
    std::string name;
    const void *dst;
    size_t bytes;
    uint64_t arg[8];  // the first words of a kernel's first argument
    Clock seen;
};
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};

std::recursive_mutex mu;
// used by the objects' start-up code, which may run before this file's
std::map<const void *, std::string> &kernel_names()
{
    static std::map<const void *, std::string> names;
    return names;
}
std::map<const void *, void *> &symbols()
{
    static std::map<const void *, void *> addresses;
    return addresses;
}
std::map<void *, size_t> blocks;
std::vector<Op> ops;
std::vector<Stream *> streams;
Stream default_stream;
Clock host;  // what host waits have covered
size_t largest = ~(size_t)0, total = ~(size_t)0, allocated = 0;
int next_capture = 0;
unsigned pause_us = 0;
bool hold = false;
std::vector<std::pair<void *, uint64_t>> held;
thread_local int call_id = 0;
float elapsed_ms = 1;
std::string json;
thread_local cudaError_t last = cudaSuccess;
thread_local cudaStreamCaptureMode thread_mode = cudaStreamCaptureModeGlobal;
thread_local std::vector<Config> configs;

cudaError_t ret(cudaError_t e)
{
    if (e != cudaSuccess)
        last = e;
    return e;
}
Stream *get(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : &default_stream; }
Event *get(cudaEvent_t e) { return reinterpret_cast<Event *>(e); }

// A call that may not be made while a stream is captured in global mode: the
// capture is lost, as in CUDA.
bool unsafe()
{
    bool hit = false;
    if (thread_mode != cudaStreamCaptureModeRelaxed)
        for (Stream *s : streams)
            if (s->capture && s->global)
                hit = s->broken = true;
    return hit;
}

void record(cudaStream_t stream, const std::string &name, const void *dst, size_t bytes, const void *arg = nullptr)
{
    Stream *s = get(stream);
    join(s->seen, host);
    s->seen[s->id]++;
    Op o{call_id, s->id, s->seen[s->id], name, dst, bytes, {}, s->seen};
    if (arg)
        memcpy(o.arg, arg, sizeof o.arg);
    ops.push_back(o);
}
void wait_all()
{
    for (Stream *s : streams)
        join(host, s->seen);
    join(host, default_stream.seen);
}

}  // namespace

extern "C" {

// ---- test controls -----------------------------------------------------------
void fake_call(int id) { call_id = id; }                    // tags the operations of this thread that follow
void fake_pause(unsigned us) { pause_us = us; }              // after every copy, so that other threads come in
void fake_hold(int on)  // keeps 8-byte results from the host, as of work that has not ended, until let go
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    hold = on != 0;
    for (const auto &[dst, word] : held)
        if (!hold)
            memcpy(dst, &word, 8);
    if (!hold)
        held.clear();
}
void fake_largest_malloc(size_t bytes) { largest = bytes; }  // larger ones fail
void fake_total(size_t bytes) { total = bytes; }             // more than that at once fails
void fake_elapsed(float ms) { elapsed_ms = ms; }
size_t fake_allocated() { return allocated; }
int fake_blocks(uint64_t *address, int most)  // of device memory
{
    int n = 0;
    for (const auto &b : blocks)
        if (n < most)
            address[n++] = (uint64_t)b.first;
    return n;
}
void fake_clear()
{
    ops.clear();
    last = cudaSuccess;
    for (Stream *s : streams)
        s->capture = 0;
}
const char *fake_ops()
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    std::ostringstream o;
    o << "[";
    for (size_t i = 0; i < ops.size(); i++) {
        const Op &p = ops[i];
        o << (i ? "," : "") << "{\"call\":" << p.call << ",\"stream\":" << p.stream << ",\"index\":" << p.index
          << ",\"name\":\"" << p.name << "\",\"dst\":" << (uint64_t)p.dst << ",\"bytes\":" << p.bytes << ",\"arg\":[";
        for (int k = 0; k < 8; k++)
            o << (k ? "," : "") << p.arg[k];
        o << "],\"seen\":{";
        bool first = true;
        for (const auto &[s, n] : p.seen) {
            o << (first ? "" : ",") << "\"" << s << "\":" << n;
            first = false;
        }
        o << "}}";
    }
    o << "]";
    json = o.str();
    return json.c_str();
}

// ---- compiler interface ------------------------------------------------------
void **__cudaRegisterFatBinary(void *) { return new void *(nullptr); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **h) { delete h; }
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *)
{
    kernel_names()[fun] = name;
}
void __cudaRegisterVar(void **, char *var, char *, const char *, int, size_t size, int, int)
{
    symbols()[var] = calloc(1, size);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s)
{
    configs.push_back({grid, block, smem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s)
{
    const Config c = configs.back();
    configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *static_cast<cudaStream_t *>(s) = c.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t s)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    record(s, kernel_names()[f], nullptr, 0, args ? args[0] : nullptr);
    return cudaSuccess;
}

// ---- device and functions ----------------------------------------------------
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int)
{
    memset(p, 0, sizeof *p);
    strcpy(p->name, "host test");
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e)
{
    return e == cudaErrorMemoryAllocation ? "out of memory" : "host test error";
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *)
{
    memset(a, 0, sizeof *a);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    return *n = 1, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) { return *p = symbols()[symbol], cudaSuccess; }

// ---- memory ------------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t bytes)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (unsafe())
        return ret(cudaErrorStreamCaptureUnsupported);
    if (bytes > largest || allocated + bytes > total)
        return ret(cudaErrorMemoryAllocation);
    *p = aligned_alloc(4096, (bytes + 4095) / 4096 * 4096);
    memset(*p, 0, bytes < (1 << 20) ? bytes : (1 << 20));
    blocks[*p] = bytes;
    allocated += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!p)
        return cudaSuccess;
    if (unsafe())
        return ret(cudaErrorStreamCaptureUnsupported);
    wait_all();
    allocated -= blocks[p];
    blocks.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) { return *p = calloc(1, bytes ? bytes : 1), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total)
{
    return *free_b = *total = (size_t)180 << 30, cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    memset(a, 0, sizeof *a);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t s)
{
    {
        std::lock_guard<std::recursive_mutex> lk(mu);
        if (hold && kind == cudaMemcpyDeviceToHost && n == 8) {
            held.push_back({dst, 0});
            memcpy(&held.back().second, src, 8);
        } else {
            memcpy(dst, src, n);
        }
        record(s, kind == cudaMemcpyHostToDevice ? "h2d" : kind == cudaMemcpyDeviceToHost ? "d2h" : "copy", dst, n);
    }
    if (pause_us)
        usleep(pause_us);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t s)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    for (size_t i = 0; i < h; i++)
        memcpy(static_cast<char *>(dst) + i * dp, static_cast<const char *>(src) + i * sp, w);
    record(s, "copy2d", dst, dp * h);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind)
{
    return memcpy(dst, src, n), cudaSuccess;
}
cudaError_t cudaMemcpy2D(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h, cudaMemcpyKind)
{
    for (size_t i = 0; i < h; i++)
        memcpy(static_cast<char *>(dst) + i * dp, static_cast<const char *>(src) + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *dst, int v, size_t n, cudaStream_t s)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    memset(dst, v, n);
    record(s, "memset", dst, n);
    return cudaSuccess;
}

// ---- streams and events ------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *out, unsigned)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    Stream *s = new Stream;
    streams.push_back(s);
    s->id = (int)streams.size();
    *out = reinterpret_cast<cudaStream_t>(s);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }  // kept: its clock may be joined later
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (unsafe())
        return ret(cudaErrorStreamCaptureUnsupported);
    join(host, get(s)->seen);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t stream, cudaEvent_t event, unsigned)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    Stream *s = get(stream);
    Event *e = get(event);
    if (s->capture && e->capture != s->capture) {
        s->broken = true;
        return ret(cudaErrorStreamCaptureIsolation);
    }
    join(s->seen, e->at);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *out, unsigned)
{
    *out = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *out) { return cudaEventCreateWithFlags(out, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete get(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    get(e)->at = get(s)->seen;
    get(e)->capture = get(s)->capture;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (unsafe())
        return ret(cudaErrorStreamCaptureUnsupported);
    join(host, get(e)->at);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = elapsed_ms, cudaSuccess; }

// ---- capture -----------------------------------------------------------------
cudaError_t cudaStreamBeginCapture(cudaStream_t stream, cudaStreamCaptureMode mode)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    Stream *s = get(stream);
    s->capture = ++next_capture;
    s->global = mode == cudaStreamCaptureModeGlobal;
    s->broken = false;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t stream, cudaGraph_t *graph)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    Stream *s = get(stream);
    s->capture = 0;
    *graph = nullptr;
    return s->broken ? ret(cudaErrorStreamCaptureInvalidated) : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *status)
{
    *status = !get(s)->capture   ? cudaStreamCaptureStatusNone
              : get(s)->broken ? cudaStreamCaptureStatusInvalidated
                                 : cudaStreamCaptureStatusActive;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *mode)
{
    const cudaStreamCaptureMode m = thread_mode;
    thread_mode = *mode;
    *mode = m;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *exec, cudaGraph_t, unsigned long long)
{
    return *exec = nullptr, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }

}  // extern "C"

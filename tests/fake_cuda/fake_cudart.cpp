// A CUDA runtime without a GPU, for tests of the host code that prepares and
// launches kernels.  Device memory is host memory, kernels do nothing, copies
// happen at the call.  Two devices.  What a test asks about is counted: launches
// and copies on a stream of a device that is not current, allocations by device,
// copies and launches not yet waited for.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>

namespace {
std::mutex mu;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
struct Stream { int device; long pending; };   // pending: work queued since the last wait
struct Event { Stream *on; };
std::set<Stream *> streams;
std::map<void *, std::pair<int, size_t>> blocks;   // device memory: its device and size
long wrong_device = 0, launches = 0, bytes_on[2] = {0, 0};
int fail_mallocs = 0, no_driver_entry = 0;
Stream default_stream{0, 0};

Stream *of(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : &default_stream; }
cudaError_t fail(cudaError_t e) { return last = e; }
void work(cudaStream_t s) {
    Stream *x = of(s);
    if (s && x->device != current) ++wrong_device;
    ++x->pending;
}
}  // namespace

// ------------------------------------------------------ what the tests read
extern "C" {
long fake_wrong_device() { return wrong_device; }
long fake_launches() { return launches; }
long fake_bytes_on(int device) { return bytes_on[device]; }
long fake_pending() {   // over all streams
    std::lock_guard<std::mutex> g(mu);
    long n = 0;
    for (Stream *x : streams) n += x->pending;
    return n;
}
void fake_fail_mallocs(int n) { fail_mallocs = n; }   // the next n
void fake_no_driver_entry(int on) { no_driver_entry = on; }
}

// ------------------------------------------------------------- the runtime
extern "C" {
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return fail(cudaErrorInvalidDevice);
    current = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *l, int *g) { *l = 0; *g = 0; return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> g(mu);
    if (fail_mallocs > 0) {
        --fail_mallocs;
        return fail(cudaErrorMemoryAllocation);
    }
    *p = std::calloc(1, n ? n : 1);
    blocks[*p] = {current, n};
    bytes_on[current] += (long)n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> g(mu);
    auto it = blocks.find(p);
    if (it == blocks.end()) return cudaSuccess;
    bytes_on[it->second.first] -= (long)it->second.second;
    blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned int) { *p = std::calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned int) { *d = h; return cudaSuccess; }

cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t st) {
    work(st);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    work(st);
    std::memset(d, v, n);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned int) {
    std::lock_guard<std::mutex> g(mu);
    Stream *x = new Stream{current, 0};
    streams.insert(x);
    *s = reinterpret_cast<cudaStream_t>(x);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned int f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::lock_guard<std::mutex> g(mu);
    streams.erase(of(s));
    delete of(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { of(s)->pending = 0; return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { of(s)->pending = 0; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { work(s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new Event{nullptr}); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned int) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { reinterpret_cast<Event *>(e)->on = of(s); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (reinterpret_cast<Event *>(e)->on) reinterpret_cast<Event *>(e)->on->pending = 0;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void *, enum cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned int) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static unsigned char array[8 << 20];
    *p = array;
    return cudaSuccess;
}
static int fake_encode(...) { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned int, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult *r) {
    *f = no_driver_entry ? nullptr : reinterpret_cast<void *>(&fake_encode);
    if (r) *r = no_driver_entry ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
    return no_driver_entry ? fail(cudaErrorSymbolNotFound) : cudaSuccess;
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
    ++launches;
    work(c->stream);
    return cudaSuccess;
}

// what the compiler's host code calls
static dim3 push_grid, push_block;
static size_t push_smem;
static cudaStream_t push_stream;
unsigned int __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, struct CUstream_st *s) {
    push_grid = g;
    push_block = b;
    push_smem = m;
    push_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
    *g = push_grid;
    *b = push_block;
    *m = push_smem;
    *static_cast<cudaStream_t *>(s) = push_stream;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(void *, dim3, dim3, void **, size_t, cudaStream_t s) {
    ++launches;
    work(s);
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(void **k, const void *f) { *k = const_cast<void *>(f); return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}

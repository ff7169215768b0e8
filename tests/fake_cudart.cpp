// A stand-in for the CUDA runtime on the host, for rp_api.cu with the launchers of
// fake_launch.cu: memory is the host's, streams and events are tokens.  fake_* set
// and read it: the failure of a chosen allocation or launch, the bytes held, what
// the launches saw.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>

namespace {
struct Fake {
    std::map<void*, size_t> held;
    size_t bytes = 0;
    long fail_malloc = -1;         // allocations until the one that fails (-1: none); then all of them
    bool fail_rest = false;
    long fail_adj = -1;            // adjoint launches until the one that fails
    cudaError_t last = cudaSuccess;
    long adj = 0, ordered = 0, sorts = 0, null_bufs = 0;
} F;
char token;
}  // namespace

extern "C" {
void fake_reset() {
    F.fail_malloc = F.fail_adj = -1;
    F.fail_rest = false;
    F.last = cudaSuccess;
    F.adj = F.ordered = F.sorts = F.null_bufs = 0;
}
void fake_fail_malloc(long after, int rest) { F.fail_malloc = after; F.fail_rest = rest; }
void fake_fail_adj(long after) { F.fail_adj = after; }
// what the launchers tell: a sort's buffers (whole: none null), an adjoint launch
// (true: it fails)
void fake_note_sort(int whole) {
    F.sorts++;
    F.null_bufs += !whole;
}
int fake_note_adj(int ordered) {
    if (F.fail_adj == 0) return 1;
    if (F.fail_adj > 0) F.fail_adj--;
    F.adj++;
    F.ordered += ordered;
    return 0;
}
long fake_bytes() { return (long)F.bytes; }
long fake_adj() { return F.adj; }
long fake_ordered() { return F.ordered; }
long fake_sorts() { return F.sorts; }
long fake_null_bufs() { return F.null_bufs; }

cudaError_t cudaMalloc(void** p, size_t n) {
    if (F.fail_malloc == 0) {
        if (!F.fail_rest) F.fail_malloc = -1;
        return F.last = cudaErrorMemoryAllocation;
    }
    if (F.fail_malloc > 0) F.fail_malloc--;
    *p = calloc(1, n ? n : 1);
    F.held[*p] = n;
    F.bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    auto it = F.held.find(p);
    if (it == F.held.end()) abort();               // not held: freed twice or never made
    F.bytes -= it->second;
    F.held.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = F.last; F.last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)&token; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)&token; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)&token; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)&token; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)&token; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
int rp_nest_maps(...) { return -5; }
}

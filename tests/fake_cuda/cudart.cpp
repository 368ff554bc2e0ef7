// A CUDA runtime that runs nothing: device memory is host memory up to a capacity, copies copy, launches are counted.
// The library's host code linked against it shows, without a GPU, what it does where device memory runs out.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>

namespace {
std::map<void *, size_t> blocks;
size_t used = 0, capacity = (size_t)1 << 40, largest = 0;
long fail_at = 0, mallocs = 0, failed = 0, launches = 0, attributes = 0, null_arguments = 0;
char handle;   // what every stream and event points at
// A graph remembers the device buffers that its batched launch was given (the first four arguments: passes, instances,
// lists, items); a replay after one of them was freed is counted.
struct Graph {
    void *buf[4];
};
Graph captured;
long stale = 0, replays = 0, fused_one = 0, fused_several = 0, fused_wrong = 0;
char kernel_one, kernel_several;   // the fused passes' kernels for launches of one item, and of several
cudaError_t last = cudaSuccess;
}  // namespace

extern "C" {

// capacity of the device; what was asked of it since the last reset
void fake_set_capacity(size_t bytes) { capacity = bytes; }
void fake_fail(long nth) { fail_at = nth; }   // the nth allocation from now on fails
size_t fake_used(void) { return used; }
long fake_count(int what) {
    return what == 0 ? mallocs : what == 1 ? failed : what == 2 ? launches : what == 3 ? attributes : what == 4 ? null_arguments : what == 5 ? stale : what == 6 ? replays : what == 7 ? fused_one
         : what == 8 ? fused_several : fused_wrong;
}
size_t fake_largest(void) { return largest; }
void fake_reset(void) { mallocs = failed = launches = attributes = null_arguments = stale = replays = fused_one = fused_several = fused_wrong = 0, largest = 0; }

cudaError_t cudaMalloc(void **p, size_t n) {
    mallocs++;
    *p = nullptr;
    if (used + n > capacity || (fail_at && --fail_at == 0)) {
        failed++;
        return last = cudaErrorMemoryAllocation;
    }
    *p = calloc(n ? n : 1, 1);
    blocks[*p] = n;
    used += n;
    largest = n > largest ? n : largest;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    const auto it = blocks.find(p);
    if (it == blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    used -= it->second;
    blocks.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
    *f = capacity > used ? capacity - used : 0;
    *t = capacity;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    if (n && (!d || !s)) return last = cudaErrorInvalidValue;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemcpy2D(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t i = 0; i < h; i++) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
    if (v || n < ((size_t)1 << 20)) memset(d, v, n);   // large buffers come zeroed and stay so
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = &handle; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)&handle; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    captured = Graph();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    *g = (cudaGraph_t) new Graph(captured);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    replays++;
    for (void *b : ((Graph *)x)->buf) stale += b && !blocks.count(b);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete (Graph *)g;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete (Graph *)x;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&handle; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { attributes++; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof *a);
    a->maxThreadsPerBlock = 512;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t) {
    launches++;
    fused_one += f == &kernel_one;
    fused_several += f == &kernel_several;
    fused_wrong += (f == &kernel_one && grid.y != 1) || (f == &kernel_several && grid.y < 2);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    memcpy(captured.buf, args[0], sizeof captured.buf);   // the batched launch
    for (void *b : captured.buf) null_arguments += !b;
    return cudaLaunchKernel(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}

// what the compiler's registration code calls
void **__cudaRegisterFatBinary(void *) { static void *h = &handle; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
char __cudaInitModule(void **) { return 0; }
static dim3 cfg_grid, cfg_block;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, cudaStream_t) {
    cfg_grid = g;
    cfg_block = b;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sm, void *st) {
    *g = cfg_grid;
    *b = cfg_block;
    *sm = 0;
    *(cudaStream_t *)st = (cudaStream_t)&handle;
    return cudaSuccess;
}

}  // extern "C"

// the fused passes' kernels are picked in translation units of their own, which are left out
namespace gsb {
static void *fused(bool several) { return several ? &kernel_several : &kernel_one; }
template <bool S> void *pick_group_f32(int, int) { return fused(S); }
template <bool S> void *pick_group3(int, int) { return fused(S); }
template <bool S> void *pick_group_ws(int, int) { return fused(S); }
template <bool S> void *pick_group128(int, int, bool) { return fused(S); }
template void *pick_group_f32<false>(int, int);
template void *pick_group_f32<true>(int, int);
template void *pick_group3<false>(int, int);
template void *pick_group3<true>(int, int);
template void *pick_group_ws<false>(int, int);
template void *pick_group_ws<true>(int, int);
template void *pick_group128<false>(int, int, bool);
template void *pick_group128<true>(int, int, bool);
}  // namespace gsb

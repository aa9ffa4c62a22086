// A CUDA runtime without a device, for host programs linked with libgeofd:
// the functions below come before the runtime library's in symbol lookup.
// Device memory is host memory under a limit, copies are copies, kernels do
// nothing but a few that the host reads results of, and what belongs to a
// device (constant memory, kernel attributes) is kept per device, so that a
// launch whose shared memory the device's attribute does not allow fails as
// it does on a GPU.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

namespace fake {
// built on first use: the library registers its kernels before main's statics
struct State {
    std::recursive_mutex mu;
    std::map<const void *, std::string> kernel_name, symbol_name;
    std::map<int, std::set<std::string>> symbols, attributes;   // set so far, by device
    std::map<std::pair<int, const void *>, size_t> smem_limit;
    std::map<void *, size_t> blocks;
    size_t in_use = 0, peak = 0, limit = ~size_t(0);
    std::map<std::string, long> launches, blocks_max;
    std::string refused;   // launches that a device would refuse
    int device_waits = 0;
    void (*on_launch)(const std::string &, void **) = nullptr;
};
inline State &st() {
    static State *s = new State;
    return *s;
}
inline thread_local int device = 0;
inline thread_local cudaError_t last = cudaSuccess;

inline cudaError_t err(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}

inline cudaError_t launch(const void *f, dim3 grid, void **args, size_t smem) {
    std::lock_guard<std::recursive_mutex> g(st().mu);
    const std::string &n = st().kernel_name[f];
    st().launches[n]++;
    if (grid.x > st().blocks_max[n]) st().blocks_max[n] = grid.x;
    const auto it = st().smem_limit.find({device, f});
    if (smem > 49152 && (it == st().smem_limit.end() || it->second < smem)) {
        st().refused += n + " on device " + std::to_string(device) + "\n";
        return err(cudaErrorInvalidValue);
    }
    if (st().on_launch) st().on_launch(n, args);
    const unsigned v = 0x44fa0000u;   // 2000.0f
    if (n.find("k_raw_stats") != n.npos) {
        struct View { const float *a[4]; int nx, nz; } *r = (View *)args[0];
        unsigned *head = *(unsigned **)args[1];
        head[4] = v;
        head[5] = ~v;
        for (int x = 0; x < r->nx; x++) (*(float **)args[2])[x] = 2000.0f;
    } else if (n.find("k_pick") != n.npos) {
        struct View { const float *a[4]; int nx, nz; } *r = (View *)args[0];
        const unsigned long long *idx = *(unsigned long long **)args[1];
        for (int k = 0; k < *(int *)args[2]; k++)
            (*(float **)args[3])[k] = r->a[idx[k] >> 60][idx[k] & ((1ull << 60) - 1)];
    } else if (n.find("k_minmax") != n.npos) {
        (*(unsigned **)args[2])[0] = (*(unsigned **)args[2])[1] = v;
    }
    return cudaSuccess;
}
}  // namespace fake

#define FAKE extern "C" __attribute__((visibility("default")))
struct FakeConfig { dim3 grid, block; size_t smem; cudaStream_t s; };
inline thread_local FakeConfig fake_config;

FAKE void **__cudaRegisterFatBinary(void *) { static void *h[1]; return h; }
FAKE void __cudaRegisterFatBinaryEnd(void **) {}
FAKE void __cudaUnregisterFatBinary(void **) {}
FAKE void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    fake::st().kernel_name[f] = name;
}
FAKE void __cudaRegisterVar(void **, char *v, char *, const char *name, int, size_t, int, int) { fake::st().symbol_name[v] = name; }
FAKE unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *s) {
    fake_config = {g, b, smem, s};
    return 0;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
    *g = fake_config.grid;
    *b = fake_config.block;
    *smem = fake_config.smem;
    *(cudaStream_t *)s = fake_config.s;
    return cudaSuccess;
}
FAKE cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
FAKE cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void **args, size_t smem, cudaStream_t) {
    return fake::launch((const void *)k, g, args, smem);
}
FAKE cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **args, size_t smem, cudaStream_t) {
    return fake::launch(f, g, args, smem);
}
FAKE cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3, void **args, size_t smem, cudaStream_t) {
    return fake::launch(f, g, args, smem);
}
FAKE cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    return fake::launch(f, c->gridDim, args, c->dynamicSmemBytes);
}
FAKE cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute, int v) {
    std::lock_guard<std::recursive_mutex> g(fake::st().mu);
    fake::st().smem_limit[{fake::device, f}] = v;
    fake::st().attributes[fake::device].insert(fake::st().kernel_name[f]);
    return cudaSuccess;
}
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int threads, size_t smem) {
    *n = (int)(233472 / (smem + 1024));
    if (*n > 65536 / (128 * threads)) *n = 65536 / (128 * threads);
    return cudaSuccess;
}
FAKE cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::recursive_mutex> g(fake::st().mu);
    if (n > fake::st().limit - fake::st().in_use) return fake::err(cudaErrorMemoryAllocation);
    if (posix_memalign(p, 512, n)) return fake::err(cudaErrorMemoryAllocation);
    memset(*p, 0, n);
    fake::st().blocks[*p] = n;
    fake::st().in_use += n;
    if (fake::st().in_use > fake::st().peak) fake::st().peak = fake::st().in_use;
    return cudaSuccess;
}
FAKE cudaError_t cudaFree(void *p) {
    std::lock_guard<std::recursive_mutex> g(fake::st().mu);
    const auto it = fake::st().blocks.find(p);
    if (it != fake::st().blocks.end()) {
        fake::st().in_use -= it->second;
        fake::st().blocks.erase(it);
        free(p);
    }
    return cudaSuccess;
}
FAKE cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = fake::st().limit - fake::st().in_use; *t = fake::st().limit; return cudaSuccess; }
FAKE cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(n, 1); return cudaSuccess; }
FAKE cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
FAKE cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
FAKE cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
FAKE cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
FAKE cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t k = 0; k < h; k++) memcpy((char *)d + k * dp, (const char *)s + k * sp, w);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
FAKE cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
FAKE cudaError_t cudaMemcpyToSymbol(const void *sym, const void *, size_t, size_t, cudaMemcpyKind) {
    std::lock_guard<std::recursive_mutex> g(fake::st().mu);
    fake::st().symbols[fake::device].insert(fake::st().symbol_name[sym]);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemcpyToSymbolAsync(const void *sym, const void *s, size_t n, size_t o, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpyToSymbol(sym, s, n, o, k);
}
FAKE cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
    std::lock_guard<std::recursive_mutex> g(fake::st().mu);
    static std::map<std::pair<int, const void *>, void *> at;
    void *&q = at[{fake::device, sym}];
    if (!q) q = calloc(64 << 20, 1);
    *p = q;
    return cudaSuccess;
}
FAKE cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
FAKE cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }
FAKE cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
FAKE cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
FAKE cudaError_t cudaDeviceSynchronize() { fake::st().device_waits++; return cudaSuccess; }
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
FAKE cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = (cudaGraph_t)1; return cudaSuccess; }
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)1; return cudaSuccess; }
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
FAKE cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 1.0f; return cudaSuccess; }
FAKE const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
FAKE cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
inline CUresult fake_encode(CUtensorMap *m, CUtensorMapDataType, cuuint32_t, void *base, const cuuint64_t *, const cuuint64_t *,
                            const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    memset(m, 0, sizeof *m);
    memcpy(m, &base, sizeof base);
    if (!base) fake::st().refused += "tensor map of a null buffer\n";
    return CUDA_SUCCESS;
}
FAKE cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned, unsigned long long,
                                                  enum cudaDriverEntryPointQueryResult *q) {
    *f = (void *)fake_encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

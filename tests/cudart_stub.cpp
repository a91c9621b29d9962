// A CUDA runtime without a GPU, preloaded before libcudart: device memory is host memory under a limit, copies and fills happen at once,
// kernels do nothing.  It serves tests of host logic: which memory a call takes, how a prompt is cut, and whether work on a stream may run before a fill that
// was queued on the default stream, and which kernels with which grids a call launches.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include <cuda.h>
#include <cuda_runtime_api.h>

static std::mutex mu;
static std::map<char*, size_t> blocks;                 // device memory
static std::map<char*, size_t> filled;                 // written on the default stream since the device was last waited for
static size_t limit = (size_t)1 << 40, used = 0, peak = 0;
static long unordered = 0;
static std::string copies;                             // bytes of every host-to-device copy on a stream
static std::map<const void*, std::string> kernels;     // host stub -> name of the kernel
static std::string launches;                           // name gx,gy,gz cluster-x,y,z, a line a launch
static int sms = 148;
static cudaError_t last = cudaSuccess;

static size_t device_range(const void* p, char** base) {
    auto it = blocks.upper_bound((char*)p);
    if (it == blocks.begin()) return 0;
    --it;
    if ((char*)p >= it->first + it->second) return 0;
    *base = it->first;
    return it->second;
}
// Work is queued on a stream that does not wait for the default one: every block that a fill may still be writing counts.
static void work_on(cudaStream_t s) { if (s) unordered += (long)filled.size(); }
static void launched(const void* f, dim3 g, dim3 c, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(mu);
    work_on(s);
    char at[96];
    snprintf(at, sizeof at, " %u,%u,%u %u,%u,%u\n", g.x, g.y, g.z, c.x, c.y, c.z);
    launches += kernels[f] + at;
}
static cudaError_t err(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }

extern "C" {
// ---- what a test asks and sets
void stub_limit(size_t bytes) { limit = bytes; }
size_t stub_used() { return used; }
size_t stub_peak() { const size_t p = peak; peak = used; return p; }
long stub_unordered() { const long n = unordered; unordered = 0; return n; }
void stub_sms(int n) { sms = n; }
const char* stub_launches() { static std::string out; out = launches; launches.clear(); return out.c_str(); }
const char* stub_copies() { static std::string out; out = copies; copies.clear(); return out.c_str(); }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(mu);
    if (used + n > limit) return err(cudaErrorMemoryAllocation);
    *p = aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    if (!*p) return err(cudaErrorMemoryAllocation);
    blocks[(char*)*p] = n; used += n;
    if (used > peak) peak = used;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lk(mu);
    auto it = blocks.find((char*)p);
    if (it == blocks.end()) return p ? err(cudaErrorInvalidValue) : cudaSuccess;
    used -= it->second; blocks.erase(it); filled.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) { *free_bytes = limit > used ? limit - used : 0; *total = limit; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) {
    std::lock_guard<std::mutex> lk(mu);
    char* base = nullptr;
    if (device_range(p, &base)) filled[base] = n;
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { if (!s) return cudaMemset(p, v, n); std::lock_guard<std::mutex> lk(mu); work_on(s); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::lock_guard<std::mutex> lk(mu); memcpy(d, s, n); filled.clear(); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    std::lock_guard<std::mutex> lk(mu);
    work_on(st);
    if (k == cudaMemcpyHostToDevice) copies += std::to_string(n) + " ";
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t i = 0; i < h; ++i) memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t st) { { std::lock_guard<std::mutex> lk(mu); work_on(st); } return cudaMemcpy2D(d, dp, s, sp, w, h, k); }

// ---- device, streams, events
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = sms; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { std::lock_guard<std::mutex> lk(mu); filled.clear(); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (!s) cudaDeviceSynchronize(); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }

// ---- kernels
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void**, size_t, cudaStream_t s) { launched(f, g, dim3(1, 1, 1), s); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    dim3 cl(1, 1, 1);
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cl = dim3(c->attrs[i].val.clusterDim.x, c->attrs[i].val.clusterDim.y, c->attrs[i].val.clusterDim.z);
    launched(f, c->gridDim, cl, c->stream);
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* handle[1]; return handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { kernels[host] = name; }
static thread_local struct { dim3 g, b; size_t smem; void* s; } config;      // between the two halves of kernel<<<>>>()
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) { config = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) { *g = config.g; *b = config.b; *smem = config.smem; *(void**)s = config.s; return cudaSuccess; }
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = strcmp(name, "cuTensorMapEncodeTiled") ? nullptr : (void*)encode;
    *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}

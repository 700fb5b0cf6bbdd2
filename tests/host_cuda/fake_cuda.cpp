// A CUDA runtime without a GPU, for tests of the library's host side: the objects of
// the library link against this one instead of cudart. Memory is host memory, copies
// are done at once, kernel launches are not run; what was asked of the device is
// written to a log, a line a call, and an allocation can be told to fail.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

std::mutex g_mu;
std::string g_log, g_copy;
std::map<void*, size_t> g_blocks;
std::map<const void*, std::string> g_kernels;     // host stub -> mangled device name
int g_fail_pitch = 0, g_fail_pool = 0, g_captures = 0;
thread_local cudaError_t t_last = cudaSuccess;
thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;
struct Push {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Push t_push;

template <typename... A>
void note(const char* fmt, A... a) {
    char b[1024];
    snprintf(b, sizeof b, fmt, a...);
    std::lock_guard<std::mutex> lk(g_mu);
    g_log += b;
    g_log += '\n';
}
cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) t_last = e;
    return e;
}
cudaError_t get(void** p, size_t bytes) {
    void* m = mmap(nullptr, bytes ? bytes : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return ret(cudaErrorMemoryAllocation);
    *p = m;
    std::lock_guard<std::mutex> lk(g_mu);
    g_blocks[m] = bytes;
    return cudaSuccess;
}
cudaError_t put(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_blocks.find(p);
    if (it == g_blocks.end()) return ret(cudaErrorInvalidValue);
    munmap(p, it->second ? it->second : 1);
    g_blocks.erase(it);
    return cudaSuccess;
}
bool fails(int& n) {
    std::lock_guard<std::mutex> lk(g_mu);
    return n > 0 && n-- > 0;
}
template <typename T>
cudaError_t handle(T* h) {
    static std::atomic<size_t> next{1};
    *h = reinterpret_cast<T>(next++ << 8);
    return cudaSuccess;
}

}  // namespace

extern "C" {

// The test's side.
const char* fake_log() {
    std::lock_guard<std::mutex> lk(g_mu);
    g_copy.swap(g_log);
    g_log.clear();
    return g_copy.c_str();
}
const char* fake_kernels() {               // mangled names, a line each
    std::lock_guard<std::mutex> lk(g_mu);
    g_copy.clear();
    for (const auto& k : g_kernels) g_copy += k.second + '\n';
    return g_copy.c_str();
}
void fake_fail(int pitch, int pool) {      // the next `pitch` image and `pool` pool allocations fail
    std::lock_guard<std::mutex> lk(g_mu);
    g_fail_pitch = pitch;
    g_fail_pool = pool;
}

// Registration and launches.
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    t_push = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = t_push.grid, *block = t_push.block, *smem = t_push.smem;
    *static_cast<cudaStream_t*>(stream) = t_push.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    // The limits that a real launch checks.
    if (grid.x > 0x7FFFFFFFu || grid.y > 65535u || grid.z > 65535u || !grid.x || !grid.y || block.x * block.y * block.z > 1024u)
        return ret(cudaErrorInvalidConfiguration);
    note("launch %s grid %u %u %u block %u smem %zu", g_kernels[fn].c_str(), grid.x, grid.y, grid.z,
         block.x * block.y * block.z, smem);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
    return cudaLaunchKernel(fn, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    memset(a, 0, sizeof *a);
    a->maxThreadsPerBlock = 1024;
    a->numRegs = 124;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 4;
    return cudaSuccess;
}

// Memory.
cudaError_t cudaMallocPitch(void** p, size_t* pitch, size_t width, size_t height) {
    if (fails(g_fail_pitch)) return ret(cudaErrorMemoryAllocation);
    *pitch = (width + 511) / 512 * 512;
    const cudaError_t e = get(p, *pitch * height);
    note("mallocpitch %p %zu mode %d", *p, *pitch * height, (int)t_mode);
    return e;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    const cudaError_t e = get(p, n);
    note("malloc %p %zu", *p, n);
    return e;
}
cudaError_t cudaFree(void* p) {
    note("free %p", p);
    return put(p);
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (fails(g_fail_pool)) return ret(cudaErrorMemoryAllocation);
    note("mallocpool %zu", n);
    return get(p, n);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return put(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return get(p, n); }
cudaError_t cudaFreeHost(void* p) { return put(p); }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
    static std::map<const void*, void*> at;
    std::lock_guard<std::mutex> lk(g_mu);
    void*& m = at[symbol];
    if (!m) m = mmap(nullptr, 64u << 20, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    *p = m;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t y = 0; y < h; ++y) memcpy((char*)d + y * dp, (const char*)s + y * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    *free_bytes = *total = (size_t)180 << 30;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { return handle(p); }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) {
    *static_cast<uint64_t*>(v) = 0;
    return cudaSuccess;
}

// Devices, streams, events, graphs.
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount            ? 148
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
         : a == cudaDevAttrMaxRegistersPerMultiprocessor ? 65536
                                                         : 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    std::swap(*m, t_mode);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) {
    *n = 0;
    return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType* t) {
    *t = cudaGraphNodeTypeKernel;
    return cudaSuccess;
}
cudaError_t cudaGraphEventRecordNodeGetEvent(cudaGraphNode_t, cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaGraphExecEventRecordNodeSetEvent(cudaGraphExec_t, cudaGraphNode_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return handle(x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"

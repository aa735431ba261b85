// A CUDA runtime on host memory, loaded in front of the real one (LD_PRELOAD),
// for tests of the engine's host code without a device: copies are memcpy,
// kernels do not run.  fake_* set what fails and count what was done.  With it
// come an operator new that can fail at the nth allocation of the arming thread
// (host allocation failures) and slow synchronisation and attribute calls
// (overlap of threads).
#include <cuda_runtime_api.h>

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <thread>

namespace {
std::mutex mu;
struct State {
    std::map<const void*, std::string> kernels;
    std::map<const void*, int> max_dynamic;  // per kernel
    std::map<std::string, int> launches, threads;  // threads: of the last launch's blocks
    std::map<void*, std::pair<size_t, bool>> blocks;  // device memory: bytes, of a pool
    std::set<void*> freed;  // blocks of at most 1 MB given back (their addresses are not used again)
};
State& st() {
    static State* s = new State;
    return *s;
}
size_t limit = size_t(8) << 30, live = 0, kept = 0;  // live: allocated; kept: freed but held by the pools
std::atomic<int> host_allocs{0}, no_pinned{0}, sync_ms{0}, attr_ms{0};
thread_local long new_countdown = 0;
thread_local bool new_fired = false;
struct Held {  // the runtime's own state: locked, and its allocations not counted
    std::lock_guard<std::mutex> lock{mu};
    long countdown = new_countdown;
    Held() { new_countdown = 0; }
    ~Held() { new_countdown = countdown; }
};
void nap(int ms) {
    if (ms) std::this_thread::sleep_for(std::chrono::milliseconds(ms));
}
cudaError_t take(void** p, size_t n, bool pooled) {
    Held held;
    const size_t reused = pooled ? std::min(n, kept) : 0;
    if (live + kept - reused + n > limit) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, n ? n : 1);
    kept -= reused;
    live += n;
    st().blocks[*p] = {n, pooled};
    return cudaSuccess;
}
cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    Held held;
    const auto b = st().blocks[p];
    st().blocks.erase(p);
    live -= b.first;
    if (b.second) kept += b.first;
    if (b.first <= (1 << 20)) st().freed.insert(p);
    else std::free(p);
    return cudaSuccess;
}
}  // namespace

void* operator new(size_t n) {
    if (new_countdown > 0 && --new_countdown == 0) {
        new_fired = true;
        throw std::bad_alloc();
    }
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
void fake_limit(size_t n) { limit = n; }
size_t fake_live() { return live; }
int fake_dangling() {  // pointers to freed blocks in live ones of at most 4 KB
    Held held;
    int n = 0;
    for (auto& b : st().blocks)
        for (size_t k = 0; b.second.first <= 4096 && k + 8 <= b.second.first; k += 8) {
            void* q;
            std::memcpy(&q, static_cast<char*>(b.first) + k, 8);
            n += (int)st().freed.count(q);
        }
    return n;
}
int fake_host_allocs() { return host_allocs; }
void fake_no_pinned(int none) { no_pinned = none; }
void fake_sync_ms(int ms) { sync_ms = ms; }
void fake_attr_ms(int ms) { attr_ms = ms; }
void fake_fail_new(long nth) { new_countdown = nth; new_fired = false; }
int fake_new_fired() { new_countdown = 0; return new_fired; }
int fake_launches(const char* part) {  // launches of kernels whose (mangled) name holds `part`
    Held held;
    int n = 0;
    for (auto& k : st().launches)
        if (k.first.find(part) != std::string::npos) n += k.second;
    return n;
}
int fake_threads(const char* part) {  // threads per block of such a kernel's last launch
    Held held;
    for (auto& k : st().threads)
        if (k.first.find(part) != std::string::npos) return k.second;
    return 0;
}
int fake_max_dynamic(const char* part) {  // the largest dynamic shared memory such a kernel is set to
    Held held;
    int n = 0;
    for (auto& k : st().kernels)
        if (k.second.find(part) != std::string::npos && st().max_dynamic.count(k.first))
            n = std::max(n, st().max_dynamic[k.first]);
    return n;
}

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    Held held;
    st().kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local dim3 call_grid, call_block;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, cudaStream_t) {
    call_grid = g;
    call_block = b;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* stream) {
    *g = call_grid;
    *b = call_block;
    *s = 0;
    *static_cast<cudaStream_t*>(stream) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3 block, void**, size_t, cudaStream_t) {
    Held held;
    st().launches[st().kernels[f]]++;
    st().threads[st().kernels[f]] = (int)(block.x * block.y * block.z);
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    *a = cudaFuncAttributes{};
    a->sharedSizeBytes = 2048;
    {
        Held held;
        a->maxDynamicSharedSizeBytes = st().max_dynamic.count(f) ? st().max_dynamic[f] : 48 * 1024;
    }
    nap(attr_ms);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    Held held;
    st().max_dynamic[f] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem, unsigned) {
    *n = std::min(512 / threads, (int)(233472 / (smem + 3072)));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
}
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
#undef cudaGetDeviceProperties
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    p->sharedMemPerBlockOptin = 232448;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char mem[16 << 20];
    *p = mem;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, false); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n, true); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return take(p, n, true); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)1; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { Held held; kept = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { Held held; kept = 0; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = limit - live - kept; *t = limit; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = nullptr;
    if (no_pinned) return cudaErrorMemoryAllocation;
    host_allocs++;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { nap(sync_ms); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
}

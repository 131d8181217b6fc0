// The scratch pool (pool.cpp) over a fake runtime of two devices: which blocks it hands out again, and to whom.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>

#include "fgpu_core.h"

static thread_local int t_device = 0;
static size_t g_room[2] = {16u << 20, 16u << 20};       // bytes left on each device
static std::map<void*, std::pair<int, size_t>> g_blocks;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > g_room[t_device]) return cudaErrorMemoryAllocation;
    g_room[t_device] -= n;
    *p = std::malloc(1);
    g_blocks[*p] = {t_device, n};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto b = g_blocks.find(p);
    if (b == g_blocks.end()) return cudaErrorInvalidValue;
    g_room[b->second.first] += b->second.second;
    g_blocks.erase(b);                                  // (the address is not used again)
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = g_room[t_device]; *t = 16u << 20; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->totalGlobalMem = 16u << 20;
    return cudaSuccess;
}
}

static int g_bad = 0;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); g_bad = 1; } } while (0)

static void* take(cudaStream_t s, size_t n, int dev = 0) {
    t_device = dev;
    void* p = nullptr;
    CHECK(fgpu::pool_malloc_bytes(s, &p, n) == cudaSuccess);
    CHECK(p && g_blocks.count(p) && g_blocks[p].first == dev);
    return p;
}

int main() {
    const cudaStream_t a = (cudaStream_t)0x1000, b = (cudaStream_t)0x2000;
    // a stream gets its own blocks again, another stream does not
    void* p = take(a, 4096);
    fgpu::pool_free(p);
    CHECK(g_blocks.count(p) == 1);
    void* q = take(b, 4096);
    CHECK(q != p);
    CHECK(take(a, 4096) == p);
    fgpu::pool_free(q);
    fgpu::pool_free(p);
    // one handle, two devices
    for (cudaStream_t s : {cudaStreamLegacy, a}) {
        void* x = take(s, 8192, 0);
        fgpu::pool_free(x);
        void* y = take(s, 8192, 1);
        CHECK(y != x);
        fgpu::pool_free(y);
        CHECK(take(s, 8192, 1) == y);
        CHECK(take(s, 8192, 0) == x);
        t_device = 1;
        fgpu::pool_free(x);                             // freed with the other device current
        fgpu::pool_free(y);
        CHECK(take(s, 8192, 0) == x);
        fgpu::pool_free(x);
    }
    // a handle that is another stream in each thread: nothing is kept
    void* t = take(cudaStreamPerThread, 4096);
    CHECK(fgpu::pool_free(t) == cudaSuccess);
    CHECK(g_blocks.count(t) == 0);
    fgpu::pool_release(a);
    fgpu::pool_release(b);
    fgpu::pool_release(cudaStreamLegacy);
    CHECK(g_blocks.empty());
    // the bound holds for each device by itself
    std::vector<void*> v;
    for (int dev : {0, 1})
        for (int k = 0; k < 8; ++k) v.push_back(take(a, 64u << 10, dev));
    for (void* x : v) fgpu::pool_free(x);
    size_t kept[2] = {0, 0};
    for (auto& x : g_blocks) kept[x.second.first] += x.second.second;
    CHECK(kept[0] > 0 && kept[0] == kept[1] && kept[0] <= (16u << 20) / 64);
    t_device = 1;
    CHECK(fgpu::pool_kept_bytes() == kept[1]);
    // an allocation that would fail gets what is kept on its device, and on no other
    t_device = 0;
    void* big = nullptr;
    CHECK(fgpu::dev_malloc_bytes(&big, 16u << 20) == cudaSuccess);
    size_t other = 0;
    for (auto& x : g_blocks)
        if (x.second.first == 1) other += x.second.second;
    CHECK(other == kept[1]);
    fgpu::pool_free(big);
    fgpu::pool_release(a);
    CHECK(g_blocks.empty());
    // given back on request, blocks handed out stay
    p = take(a, 4096);
    q = take(a, 8192);
    fgpu::pool_free(p);
    fgpu::pool_trim(b);
    CHECK(g_blocks.count(p) == 1 && fgpu::pool_kept_bytes() == 4096);
    fgpu::pool_trim(a);
    CHECK(g_blocks.count(p) == 0 && g_blocks.count(q) == 1 && fgpu::pool_kept_bytes() == 0);
    fgpu::pool_free(q);
    CHECK(take(a, 8192) == q);
    fgpu::pool_free(q);
    fgpu::pool_release(a);
    // a block still handed out when its stream goes is freed for good
    p = take(a, 4096);
    fgpu::pool_release(a);
    fgpu::pool_free(p);
    CHECK(g_blocks.empty());
    return g_bad;
}

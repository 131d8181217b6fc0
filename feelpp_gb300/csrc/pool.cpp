// Device scratch kept between calls.
//
// A solve or an AMG set-up allocates and frees a few hundred work arrays; cudaMalloc and cudaFree take tens
// of microseconds each (14 of the 52 ms of an AMG set-up and solve at P2 48^3), and cudaFree waits for the
// device. Freed blocks are kept per device and stream instead and handed out again in stream order: a block
// freed while its kernels are still queued on its stream is only reused by later work on the same stream. (Work
// on another stream has to be joined before the block is freed.) The handle alone does not name a stream:
// cudaStreamLegacy is one handle for a stream of every device (the key holds the device), and cudaStreamPerThread
// one for a stream of every thread (its blocks are not kept: any thread may free them).
//
// Bounded: at most a sixty-fourth of a device's memory is kept (4.3 GB; CG + AMG at P2 48^3 keeps 1.3 GB, at P3 40^3
// 3.4), the rest goes back to the driver at once, and pool_trim gives back what is kept for a stream; a
// context gives its stream's blocks back when it is destroyed; and an allocation that fails, here or in
// dev_malloc, is tried again after everything kept has been given back. Page-locked host blocks (a few
// kilobytes for scalars that are read back) are kept in the same way, at most 1 MB. All functions may be
// called from several threads.
#include <algorithm>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "fgpu_core.h"

namespace fgpu {

namespace {

typedef std::pair<int, cudaStream_t> Key;                                  // device, stream
struct Block {
    Key key;
    size_t bytes;
};
struct Device {
    size_t kept = 0, limit = 0;      // bytes
};

std::mutex g_mutex;
std::unordered_map<void*, Block> g_live;                                   // handed out
std::map<Key, std::multimap<size_t, void*>> g_kept;                        // free, by size
std::map<int, Device> g_device;
std::multimap<size_t, void*> g_pinned;                                     // free page-locked blocks
std::unordered_map<void*, size_t> g_pinned_live;
size_t g_pinned_bytes = 0;
constexpr size_t kPinnedLimit = (size_t)1 << 20;

void give_back(std::vector<void*>& blocks) {
    for (void* p : blocks) cudaFree(p);
}

int current_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}

// everything kept on a device, out of the lists (the caller frees it without the lock)
std::vector<void*> take_all(int dev) {
    std::vector<void*> out;
    std::lock_guard<std::mutex> lock(g_mutex);
    for (auto s = g_kept.begin(); s != g_kept.end();) {
        if (s->first.first != dev) { ++s; continue; }
        for (auto& b : s->second) out.push_back(b.second);
        s = g_kept.erase(s);
    }
    g_device[dev].kept = 0;
    return out;
}

}  // namespace

cudaError_t dev_malloc_bytes(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    std::vector<void*> kept = take_all(current_device());
    if (kept.empty()) return e;
    cudaGetLastError();
    give_back(kept);
    return cudaMalloc(p, bytes);
}

cudaError_t pool_malloc_bytes(cudaStream_t stream, void** p, size_t bytes) {
    bytes = (std::max<size_t>(bytes, 1) + 511) & ~(size_t)511;
    if (stream == cudaStreamPerThread) return dev_malloc_bytes(p, bytes);
    const Key key(current_device(), stream);
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto s = g_kept.find(key);
        if (s != g_kept.end()) {
            auto b = s->second.lower_bound(bytes);
            if (b != s->second.end() && b->first <= bytes + bytes / 4 + 4096) {      // little is wasted
                *p = b->second;
                g_live[*p] = Block{key, b->first};
                g_device[key.first].kept -= b->first;
                s->second.erase(b);
                return cudaSuccess;
            }
        }
    }
    const cudaError_t e = dev_malloc_bytes(p, bytes);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mutex);
        g_live[*p] = Block{key, bytes};
    }
    return e;
}

cudaError_t pool_free(void* p) {
    if (!p) return cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto b = g_live.find(p);
        if (b != g_live.end()) {
            const Block blk = b->second;
            g_live.erase(b);
            Device& d = g_device[blk.key.first];
            if (d.limit == 0) {
                cudaDeviceProp prop{};
                d.limit = cudaGetDeviceProperties(&prop, blk.key.first) == cudaSuccess ? std::max<size_t>(prop.totalGlobalMem / 64, 1) : 1;
            }
            if (d.kept + blk.bytes <= d.limit) {
                g_kept[blk.key].emplace(blk.bytes, p);
                d.kept += blk.bytes;
                return cudaSuccess;
            }
        }
    }
    return cudaFree(p);
}

// bytes kept on the current device (dev_malloc can have them)
size_t pool_kept_bytes() {
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(g_mutex);
    return g_device[dev].kept;
}

// the blocks kept for a stream, back to the driver
static void take_stream(cudaStream_t stream, std::vector<void*>& out) {
    for (auto s = g_kept.begin(); s != g_kept.end();) {
        if (s->first.second != stream) { ++s; continue; }
        for (auto& b : s->second) {
            out.push_back(b.second);
            g_device[s->first.first].kept -= b.first;
        }
        s = g_kept.erase(s);
    }
}
void pool_trim(cudaStream_t stream) {
    std::vector<void*> out;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        take_stream(stream, out);
    }
    give_back(out);
}
// the same for a stream that goes away; blocks still handed out are freed for good when they come back
void pool_release(cudaStream_t stream) {
    std::vector<void*> out;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        take_stream(stream, out);
        for (auto b = g_live.begin(); b != g_live.end();) {
            if (b->second.key.second == stream) b = g_live.erase(b);
            else ++b;
        }
    }
    give_back(out);
}

cudaError_t pinned_malloc_bytes(void** p, size_t bytes) {
    bytes = (std::max<size_t>(bytes, 1) + 4095) & ~(size_t)4095;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto b = g_pinned.find(bytes);
        if (b != g_pinned.end()) {
            *p = b->second;
            g_pinned_live[*p] = bytes;
            g_pinned_bytes -= bytes;
            g_pinned.erase(b);
            return cudaSuccess;
        }
    }
    const cudaError_t e = cudaMallocHost(p, bytes);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mutex);
        g_pinned_live[*p] = bytes;
    }
    return e;
}

void pinned_free(void* p) {
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto b = g_pinned_live.find(p);
        if (b != g_pinned_live.end()) {
            const size_t bytes = b->second;
            g_pinned_live.erase(b);
            if (g_pinned_bytes + bytes <= kPinnedLimit) {
                g_pinned.emplace(bytes, p);
                g_pinned_bytes += bytes;
                return;
            }
        }
    }
    cudaFreeHost(p);
}

}  // namespace fgpu

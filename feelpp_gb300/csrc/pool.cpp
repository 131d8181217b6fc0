// Device scratch kept between calls.
//
// A solve or an AMG set-up allocates and frees a few hundred work arrays; cudaMalloc and cudaFree take tens
// of microseconds each (14 of the 52 ms of an AMG set-up and solve at P2 48^3), and cudaFree waits for the
// device. Freed blocks are kept per stream instead and handed out again in stream order: a block freed while
// its kernels are still queued on its stream is only reused by later work on the same stream. (Work on
// another stream has to be joined before the block is freed.)
//
// Bounded: at most a sixteenth of the device's memory is kept, the rest goes back to the driver at once; a
// context gives its stream's blocks back when it is destroyed; and an allocation that fails, here or in
// dev_malloc, is tried again after everything kept has been given back. Page-locked host blocks (a few
// kilobytes for scalars that are read back) are kept in the same way, at most 1 MB. All functions may be
// called from several threads.
#include <algorithm>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "fgpu_core.h"

namespace fgpu {

namespace {

struct Block {
    cudaStream_t stream;
    size_t bytes;
};

std::mutex g_mutex;
std::unordered_map<void*, Block> g_live;                                   // handed out
std::map<cudaStream_t, std::multimap<size_t, void*>> g_kept;               // free, per stream, by size
size_t g_kept_bytes = 0, g_limit = 0;
std::multimap<size_t, void*> g_pinned;                                     // free page-locked blocks
std::unordered_map<void*, size_t> g_pinned_live;
size_t g_pinned_bytes = 0;
constexpr size_t kPinnedLimit = (size_t)1 << 20;

void give_back(std::vector<void*>& blocks) {
    for (void* p : blocks) cudaFree(p);
}

// everything kept, out of the lists (the caller frees it without the lock)
std::vector<void*> take_all() {
    std::vector<void*> out;
    std::lock_guard<std::mutex> lock(g_mutex);
    for (auto& s : g_kept)
        for (auto& b : s.second) out.push_back(b.second);
    g_kept.clear();
    g_kept_bytes = 0;
    return out;
}

}  // namespace

cudaError_t dev_malloc_bytes(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    std::vector<void*> kept = take_all();
    if (kept.empty()) return e;
    cudaGetLastError();
    give_back(kept);
    return cudaMalloc(p, bytes);
}

cudaError_t pool_malloc_bytes(cudaStream_t stream, void** p, size_t bytes) {
    bytes = (std::max<size_t>(bytes, 1) + 511) & ~(size_t)511;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto s = g_kept.find(stream);
        if (s != g_kept.end()) {
            auto b = s->second.lower_bound(bytes);
            if (b != s->second.end() && b->first <= bytes + bytes / 4 + 4096) {      // little is wasted
                *p = b->second;
                g_live[*p] = Block{stream, b->first};
                g_kept_bytes -= b->first;
                s->second.erase(b);
                return cudaSuccess;
            }
        }
    }
    const cudaError_t e = dev_malloc_bytes(p, bytes);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mutex);
        g_live[*p] = Block{stream, bytes};
    }
    return e;
}

cudaError_t pool_free(void* p) {
    if (!p) return cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto b = g_live.find(p);
        if (b != g_live.end()) {
            if (g_limit == 0) {
                size_t free_b = 0, total_b = 0;
                g_limit = cudaMemGetInfo(&free_b, &total_b) == cudaSuccess ? std::max<size_t>(total_b / 16, 1) : 1;
            }
            const Block blk = b->second;
            g_live.erase(b);
            if (g_kept_bytes + blk.bytes <= g_limit) {
                g_kept[blk.stream].emplace(blk.bytes, p);
                g_kept_bytes += blk.bytes;
                return cudaSuccess;
            }
        }
    }
    return cudaFree(p);
}

// the blocks kept for a stream that goes away; blocks still handed out are freed for good when they come back
void pool_release(cudaStream_t stream) {
    std::vector<void*> out;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto s = g_kept.find(stream);
        if (s != g_kept.end()) {
            for (auto& b : s->second) {
                out.push_back(b.second);
                g_kept_bytes -= b.first;
            }
            g_kept.erase(s);
        }
        for (auto b = g_live.begin(); b != g_live.end();) {
            if (b->second.stream == stream) b = g_live.erase(b);
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

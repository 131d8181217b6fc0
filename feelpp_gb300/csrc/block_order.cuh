// Rows of a block in the order of their lengths, so that the lanes of a warp run alike: a counting sort in
// shared memory, decided anew in each launch. The order of rows of one class is not fixed; callers do not
// let it into their results.
#pragma once
#include <cstdint>

namespace fgpu {

template <int ROWS>
struct BlockOrder {
    int bins[32];
    uint16_t row[ROWS];
};

// The local row that comes t-th, longest class first; every thread calls, threads t < ROWS bring the class
// 0 .. 31 of row t (longer: larger) and receive a row. Blocks of at least 32 threads.
template <int ROWS>
__device__ __forceinline__ int block_order(BlockOrder<ROWS>& s, int cls) {
    const int t = threadIdx.x;
    __syncthreads();                                 // the last use of s is over
    if (t < 32) s.bins[t] = 0;
    __syncthreads();
    int place = 0;
    if (t < ROWS) place = atomicAdd(&s.bins[31 - cls], 1);
    __syncthreads();
    if (t < 32) {
        int x = s.bins[t];
        const int v = x;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (t >= o) x += y;
        }
        s.bins[t] = x - v;
    }
    __syncthreads();
    if (t < ROWS) s.row[s.bins[31 - cls] + place] = (uint16_t)t;
    __syncthreads();
    return t < ROWS ? s.row[t] : 0;
}

}  // namespace fgpu

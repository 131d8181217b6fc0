// Device set-up of the smoothed-aggregation hierarchy (the default of fgpu_amg_create).
//
// The construction of the host set-up (amg_setup.cpp: Vanek, Mandel, Brezina 1996; PETSc PCGAMG "agg"
// options of the reference, feelpp/feel/feelalg/preconditionerpetsc.cpp:2229-2330), every step on the
// device (but the QR of a near null space's aggregates), and every floating-point result formed in the
// host set-up's order with the same roundings, so that the device levels equal the host levels bit for bit:
//   * diagonal and strength graph: a row kernel marks |a_ij| > theta sqrt(|a_ii a_jj|) (j != i,
//     a_ij != 0); unless the graph is its own transpose, the transpose is built by counting, a scan and a
//     fill, each row sorted, and the two sorted lists merged per row (the symmetrised graph);
//   * aggregation: the host set-up's rounds of a distance-2 independent set (roots), then roots'
//     neighbours, then the rest by their first aggregated neighbour, each step a kernel over the nodes;
//   * lambda_max(D^-1 A): 12 Lanczos steps on D^-1/2 A D^-1/2 from the host set-up's start vector, rows and
//     dot products summed in a fixed partition that both set-ups share (four partial sums per row, 128 per
//     chunk of 1024 rows, 128 over the chunks), the scalars on the device until the end, the tridiagonal's
//     largest eigenvalue by the host's Sturm bisection;
//   * P0(i, agg(i)) = 1/sqrt(|agg|), A P0, and P = P0 - omega D^-1 (A P0) merged row by row;
//   * R = P^T by counting, a scan, a fill and a per-row sort;
//   * sparse products A P0, A P and R (A P): a group of lanes per row of the left factor takes its entries
//     in order, the lanes beside one another on the distinct columns of the entry's right row, so that
//     every output entry is the host's sequential sum; columns in a shared-memory hash table per row,
//     sorted and written at the end. Rows with more distinct columns than the table holds are listed and
//     redone with a larger one. A P0 of a constant near null space has one thread per row.
// Levels of at most 512 rows, and any level with a row beyond the kernels' staging capacity, go to
// the host set-up for the rest of the hierarchy (the results are the same either way).
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <memory>
#include <string>
#include <thread>
#include <vector>

#include "fgpu_core.h"
#include "ld_stream.cuh"
#include "scan.cuh"

namespace fgpu {

AmgDevCsr::AmgDevCsr(AmgDevCsr&& o) noexcept { *this = std::move(o); }
AmgDevCsr& AmgDevCsr::operator=(AmgDevCsr&& o) noexcept {
    if (this != &o) {
        std::swap(nrows, o.nrows); std::swap(ncols, o.ncols); std::swap(nnz, o.nnz);
        std::swap(ia, o.ia); std::swap(ja, o.ja); std::swap(a, o.a); std::swap(own, o.own);
    }
    return *this;
}
AmgDevCsr::~AmgDevCsr() {
    if (own) { pool_free(ia); pool_free(ja); pool_free(a); }
}

namespace {

constexpr int kStOverflow = 1;               // a row beyond a kernel's staging capacity
constexpr int kStDiag = 2;                   // a non-positive diagonal entry
constexpr int64_t kLanczosChunk = 1024;      // rows per partial sum (the host set-up's partition)
constexpr int kLanczosSteps = 12;
// Levels this small continue on the host: below it only the coarsest levels are left, whose time is the
// launches (a level takes about 60). P2 24^3, level 1 of 1455 rows: 3.9 ms on the host, 1.2 on the device.
constexpr int64_t kHandoffRows = 512;
constexpr int kSortMax = 16384;              // longest row sorted by seg_sort_kernel
constexpr int kNumBins = 4;
constexpr int kBins[kNumBins] = {256, 1024, 2048, 8192};  // hash table sizes of whole warps (at most half full)
constexpr int kBinLog[kNumBins] = {8, 10, 11, 13};
constexpr int64_t kPadBytes = (int64_t)2 << 30;   // largest padded form of a product
constexpr int64_t kGroupRows = 4096;          // products with fewer rows take a warp per row

int grid_rows(int64_t n, int per_block, int cap = 152 * 16) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + per_block - 1) / per_block, cap));
}

struct Work {                                // device scratch returned to the pool at scope exit
    cudaStream_t stream;
    std::vector<void*> ptrs;
    explicit Work(fgpu_ctx* ctx) : stream(ctx->stream) {}
    Work(const Work&) = delete;
    Work& operator=(const Work&) = delete;
    ~Work() { for (void* p : ptrs) pool_free(p); }
    template <typename T>
    T* get(int64_t n) {
        void* p = nullptr;
        if (pool_malloc(stream, &p, std::max<int64_t>(n, 1) * sizeof(T)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
};

#define DEV_TRY(call)                                                                                         \
    do {                                                                                                      \
        const cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess) { ctx->err = std::string("gamg device set-up: ") + cudaGetErrorString(e_); return FGPU_ERR_CUDA; } \
    } while (0)
#define DEV_ALLOC(ok)                                                                                         \
    do {                                                                                                      \
        if (!(ok)) { ctx->err = "gamg device set-up: device allocation failed"; return FGPU_ERR_ALLOC; }    \
    } while (0)

int alloc_csr(fgpu_ctx* ctx, AmgDevCsr& C, int64_t nrows, int64_t ncols, int64_t nnz) {
    C = AmgDevCsr();
    C.nrows = nrows;
    C.ncols = ncols;
    C.nnz = nnz;
    DEV_TRY(pool_malloc(ctx->stream, &C.ia, (nrows + 1) * sizeof(int64_t)));
    DEV_TRY(pool_malloc(ctx->stream, &C.ja, std::max<int64_t>(nnz, 1) * sizeof(int32_t)));
    DEV_TRY(pool_malloc(ctx->stream, &C.a, std::max<int64_t>(nnz, 1) * sizeof(double)));
    return FGPU_OK;
}

int read_status(fgpu_ctx* ctx, const int* d_status, int* h) {
    DEV_TRY(cudaMemcpyAsync(h, d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    DEV_TRY(cudaStreamSynchronize(ctx->stream));
    return FGPU_OK;
}

// ---------------------------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------------------------

// diagonal (the last stored (i, i) entry, as the host's `diagonal`); flags a non-positive one
__global__ void diag_kernel(int64_t n, const int64_t* __restrict__ ia, const int32_t* __restrict__ ja, const double* __restrict__ a,
                            double* __restrict__ d, int* __restrict__ status) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double v = 0.0;
        for (int64_t p = ia[i]; p < ia[i + 1]; ++p)
            if (ja[p] == i) v = a[p];
        d[i] = v;
        if (!(v > 0.0)) atomicOr(status, kStDiag);
    }
}

// strong couplings of each row: counts (out == nullptr) or columns in row order at off[i]
__global__ void strong_kernel(int64_t n, const int64_t* __restrict__ ia, const int32_t* __restrict__ ja, const double* __restrict__ a,
                              const double* __restrict__ d, double theta, uint32_t* __restrict__ cnt, const uint32_t* __restrict__ off,
                              int32_t* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t k = 0;
        for (int64_t p = ia[i]; p < ia[i + 1]; ++p) {
            const int32_t j = ja[p];
            const double v = a[p];
            if (j == i || v == 0.0) continue;
            // theta = 0 (the default): every nonzero coupling is strong (0 * sqrt of the positive, finite
            // diagonal product is 0), without the diagonal loads and the square root
            if (theta == 0.0 || fabs(v) > theta * sqrt(fabs(__dmul_rn(d[i], d[j])))) {
                if (out) out[off[i] + k] = j;
                ++k;
            }
        }
        if (cnt) cnt[i] = k;
    }
}

// column counts of a list of column indices
__global__ void col_count_kernel(int64_t nnz, const int32_t* __restrict__ col, uint32_t* __restrict__ cnt) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nnz; q += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(cnt + col[q], 1u);
}

// transpose fill: entry (i, col[q]) goes to row col[q] of the transpose (positions by cursors; the
// rows are sorted afterwards). Row pointers of the source in 32-bit (off32) or 64-bit (off64) form.
__global__ void transpose_fill_kernel(int64_t n, const uint32_t* __restrict__ off32, const int64_t* __restrict__ off64,
                                      const int32_t* __restrict__ col, const double* __restrict__ val, uint32_t* __restrict__ cursor,
                                      int32_t* __restrict__ oj, double* __restrict__ oa) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = off64 ? off64[i] : off32[i], e = off64 ? off64[i + 1] : off32[i + 1];
        for (int64_t q = b; q < e; ++q) {
            const uint32_t t = atomicAdd(cursor + col[q], 1u);
            oj[t] = (int32_t)i;
            if (val) oa[t] = val[q];
        }
    }
}

// each row's keys (and values) sorted by key: one warp per row, bitonic sort in shared memory (cap
// entries per warp)
__global__ void __launch_bounds__(128) seg_sort_kernel(int64_t n, const uint32_t* __restrict__ off32, const int64_t* __restrict__ off64,
                                                       int cap, int32_t* __restrict__ key, double* __restrict__ val,
                                                       int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char ss_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    double* sv = reinterpret_cast<double*>(ss_smem) + (size_t)warp * cap;
    int32_t* sk = reinterpret_cast<int32_t*>(ss_smem + (val ? (size_t)warps * cap * 8 : 0)) + (size_t)warp * cap;
    for (int64_t r = (int64_t)blockIdx.x * warps + warp; r < n; r += (int64_t)gridDim.x * warps) {
        const int64_t b = off64 ? off64[r] : off32[r], e = off64 ? off64[r + 1] : off32[r + 1];
        const int len = (int)(e - b);
        if (len <= 1) continue;
        if (len > cap) {
            if (lane == 0) atomicOr(status, kStOverflow);
            continue;
        }
        int P = 1;
        while (P < len) P <<= 1;
        for (int k = lane; k < P; k += 32) {
            sk[k] = k < len ? key[b + k] : INT32_MAX;
            if (val) sv[k] = k < len ? val[b + k] : 0.0;
        }
        __syncwarp();
        for (int size = 2; size <= P; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int k = lane; k < P; k += 32) {
                    const int l = k ^ stride;
                    if (l > k) {
                        const bool up = (k & size) == 0;
                        const int32_t x = sk[k], y = sk[l];
                        if ((x > y) == up) {
                            sk[k] = y;
                            sk[l] = x;
                            if (val) {
                                const double t = sv[k];
                                sv[k] = sv[l];
                                sv[l] = t;
                            }
                        }
                    }
                }
                __syncwarp();
            }
        for (int k = lane; k < len; k += 32) {
            key[b + k] = sk[k];
            if (val) val[b + k] = sv[k];
        }
        __syncwarp();
    }
}

// longest row of a CSR offset array (32- or 64-bit)
__global__ void max_row_kernel(int64_t n, const uint32_t* __restrict__ off32, const int64_t* __restrict__ off64,
                               unsigned long long* __restrict__ out) {
    unsigned long long m = 0;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
        m = max(m, (unsigned long long)(off64 ? off64[r + 1] - off64[r] : off32[r + 1] - off32[r]));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// union of two sorted rows (count when out == nullptr)
__global__ void merge_kernel(int64_t n, const uint32_t* __restrict__ pa, const int32_t* __restrict__ ja_, const uint32_t* __restrict__ pb,
                             const int32_t* __restrict__ jb, uint32_t* __restrict__ cnt, const uint32_t* __restrict__ off,
                             int32_t* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t a = pa[i], b = pb[i], k = 0;
        const uint32_t ae = pa[i + 1], be = pb[i + 1];
        while (a < ae || b < be) {
            int32_t v;
            if (b >= be || (a < ae && ja_[a] < jb[b])) v = ja_[a++];
            else if (a >= ae || jb[b] < ja_[a]) v = jb[b++];
            else { v = ja_[a++]; ++b; }
            if (out) out[off[i] + k] = v;
            ++k;
        }
        if (cnt) cnt[i] = k;
    }
}

// *asym = 1 unless every (i, j) of the graph has its (j, i): eight lanes per row, each a search of i in the
// sorted row j. A graph that is its own transpose is the symmetrised graph already, and neither the transpose
// nor its sort and merge are needed. P2 48^3 (24.8 M couplings): 202 us in place of 1300.
__global__ void __launch_bounds__(256) symmetric_kernel(int64_t n, const uint32_t* __restrict__ sp, const int32_t* __restrict__ sj,
                                                        int* __restrict__ asym) {
    const int sub = threadIdx.x & 7;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3; i < n; i += ((int64_t)gridDim.x * blockDim.x) >> 3) {
        const uint32_t e = sp[i + 1];
        bool miss = false;
        for (uint32_t q = sp[i] + sub; q < e; q += 8) {
            const int32_t j = sj[q];
            uint32_t lo = sp[j], hi = sp[j + 1];
            while (lo < hi) {                        // the first column not below i
                const uint32_t mid = lo + ((hi - lo) >> 1);
                if (sj[mid] < (int32_t)i) lo = mid + 1;
                else hi = mid;
            }
            miss |= lo >= sp[j + 1] || sj[lo] != (int32_t)i;
        }
        if (miss) *asym = 1;
    }
}

// Lanczos steps. The scalars stay on the device: al[k], be[k], the number of steps done and the stop flag
// of a breakdown, after which the kernels do nothing.
struct LanczosScalars {
    double al[kLanczosSteps], be[kLanczosSteps], norm;
    int steps, stop;
    unsigned int ticket;
};
// w_i = s_i sum_p a_p u_j, four lanes per row: lane l sums the entries congruent to l mod 4, then
// (0 + 2) + (1 + 3). Bound: the FP64 pipe, which an instruction occupies for the whole warp: rows in the
// order of their lengths (windows of 256, like the smoother's layout) keep the warp's eight rows alike,
// and u = s v is formed once, not in each entry. P2 48^3 (25.8 M entries of rows of 24 to 65): a thread
// per row 378 us, four lanes in row order 345 (half the lanes idle), by length 188.
__global__ void __launch_bounds__(256) lanczos_spmv_kernel(int64_t n, const int64_t* __restrict__ ia, const int32_t* __restrict__ ja,
                                                           const double* __restrict__ a, const int32_t* __restrict__ perm,
                                                           const double* __restrict__ s, const double* __restrict__ u,
                                                           double* __restrict__ w, const LanczosScalars* __restrict__ sc) {
    if (sc->stop) return;
    const int sub = threadIdx.x & 3;
    const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 2;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 2; __any_sync(0xffffffffu, r < n); r += step) {
        double acc = 0.0;
        int32_t i = 0;
        if (r < n) {
            i = perm[r];
            const int64_t e = ia[i + 1];
            int64_t p = ia[i] + sub;
            for (; p + 4 < e; p += 8) {
                const int32_t j0 = __ldg(ja + p), j1 = __ldg(ja + p + 4);
                const double a0 = ld_stream(a + p), a1 = ld_stream(a + p + 4);
                const double u0 = u[j0], u1 = u[j1];
                acc = __dadd_rn(acc, __dmul_rn(a0, u0));
                acc = __dadd_rn(acc, __dmul_rn(a1, u1));
            }
            if (p < e) acc = __dadd_rn(acc, __dmul_rn(ld_stream(a + p), u[__ldg(ja + p)]));
        }
        acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
        acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
        if (r < n && sub == 0) w[i] = __dmul_rn(s[i], acc);
    }
}
// the sum of 128 partial sums, one per thread, in the host set-up's order
__device__ double lanczos_tree(double t, double* sw) {
    for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = t;
    __syncthreads();
    t = __dadd_rn(__dadd_rn(sw[0], sw[1]), __dadd_rn(sw[2], sw[3]));
    __syncthreads();
    return t;
}
// the sum over the blocks of a grid of the sums over their threads; true on the thread that has it in sw[0]
__device__ bool lanczos_sum(double t, double* partial, LanczosScalars* sc, double* sw, bool* last) {
    t = lanczos_tree(t, sw);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = t;
        __threadfence();
        *last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!*last) return false;
    __threadfence();
    t = 0.0;
    for (int c = threadIdx.x; c < (int)gridDim.x; c += 128) t = __dadd_rn(t, __ldcg(partial + c));
    t = lanczos_tree(t, sw);
    if (threadIdx.x != 0) return false;
    sc->ticket = 0;
    sw[0] = t;
    return true;
}
// the start vector x (amg_lanczos_entry) and |x|: its recurrence applies X (h ^= h >> 33, its own inverse),
// a product with C and X in turn, so that the i-th state is X(C^i X(h_0)) and every entry can be formed by
// itself (on the host, as the one serial chain, it took 3 of the estimate's 6 ms at 0.9 M rows)
__global__ void __launch_bounds__(128) lanczos_random_kernel(int64_t n, double* __restrict__ v, double* __restrict__ partial,
                                                             LanczosScalars* sc) {
    __shared__ double sw[4];
    __shared__ bool last;
    const int64_t r0 = blockIdx.x * kLanczosChunk, r1 = min(n, r0 + kLanczosChunk);
    uint64_t p = amg_lanczos_power((uint64_t)(r0 + threadIdx.x + 1));
    const uint64_t p128 = amg_lanczos_power(128);
    double t = 0.0;
    for (int64_t i = r0 + threadIdx.x; i < r1; i += 128, p *= p128) {
        const double x = amg_lanczos_entry(p);
        v[i] = x;
        t = __dadd_rn(t, __dmul_rn(x, x));
    }
    if (lanczos_sum(t, partial, sc, sw, &last)) sc->norm = __dsqrt_rn(sw[0]);
}
// v = x / |x| (the start vector), vold = 0, s = 1/sqrt(d), u = s v
__global__ void lanczos_start_kernel(int64_t n, const double* __restrict__ d, double* __restrict__ s, double* __restrict__ v,
                                     double* __restrict__ vold, double* __restrict__ u, const LanczosScalars* __restrict__ sc) {
    const double norm = sc->norm;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double si = d[i] > 0.0 ? __ddiv_rn(1.0, __dsqrt_rn(d[i])) : 0.0, vi = __ddiv_rn(v[i], norm);
        s[i] = si;
        v[i] = vi;
        vold[i] = 0.0;
        u[i] = __dmul_rn(si, vi);
    }
}
// UPDATE: w -= al_k v + be_(k-1) vold, then w.w and be_k; else w.v and al_k. A block per chunk of 1024 rows,
// thread t the rows congruent to t mod 128; the last block to finish adds the chunks' sums in the same way.
// (One thread adding a chunk's products in row order took 62 us of a dot product at 0.9 M rows, and the
// scalar went through the host; now 12 to 16, 20 with the update. P2 48^3: the estimate's steps 9.2 -> 3.1 ms.)
template <bool UPDATE>
__global__ void __launch_bounds__(128) lanczos_dot_kernel(int64_t n, int k, const double* __restrict__ v, const double* __restrict__ vold,
                                                          double* __restrict__ w, double* __restrict__ partial, LanczosScalars* sc) {
    __shared__ double sw[4];
    __shared__ bool last;
    if (sc->stop) return;
    const double al = UPDATE ? sc->al[k] : 0.0, be = UPDATE && k > 0 ? sc->be[k - 1] : 0.0;
    const int64_t r0 = blockIdx.x * kLanczosChunk, r1 = min(n, r0 + kLanczosChunk);
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < (int)(kLanczosChunk / 128); ++q) {
        const int64_t i = r0 + q * 128 + threadIdx.x;
        if (i < r1) {
            double x = w[i];
            const double vi = v[i];
            if (UPDATE) {
                x = __dsub_rn(x, __dadd_rn(__dmul_rn(al, vi), __dmul_rn(be, vold[i])));
                w[i] = x;
            }
            t = __dadd_rn(t, __dmul_rn(x, UPDATE ? x : vi));
        }
    }
    if (lanczos_sum(t, partial, sc, sw, &last)) {
        t = sw[0];
        if (UPDATE) {
            const double b = __dsqrt_rn(t);
            sc->be[k] = b;
            sc->steps = k + 1;
            if (b < 1e-14 * fabs(al)) sc->stop = 1;
        } else {
            sc->al[k] = t;
        }
    }
}
// vold = v; v = w / be_k; u = s v
__global__ void lanczos_next_kernel(int64_t n, int k, const double* __restrict__ s, const double* __restrict__ w, double* __restrict__ v,
                                    double* __restrict__ vold, double* __restrict__ u, const LanczosScalars* __restrict__ sc) {
    if (sc->stop) return;
    const double b = sc->be[k];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        vold[i] = v[i];
        const double x = __ddiv_rn(w[i], b);
        v[i] = x;
        u[i] = __dmul_rn(s[i], x);
    }
}

// tentative prolongator rows: one entry (agg_i, s0[agg_i]) where agg_i >= 0
__global__ void p0_count_kernel(int64_t n, const int32_t* __restrict__ agg, uint32_t* __restrict__ cnt) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        cnt[i] = agg[i] >= 0 ? 1u : 0u;
}
__global__ void p0_fill_kernel(int64_t n, const int32_t* __restrict__ agg, const double* __restrict__ s0, const uint32_t* __restrict__ off,
                               int64_t* __restrict__ ia, int32_t* __restrict__ ja, double* __restrict__ a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
        ia[i] = off[i];
        if (i < n && agg[i] >= 0) {
            ja[off[i]] = agg[i];
            a[off[i]] = s0[agg[i]];
        }
    }
}

// P = P0 - omega D^-1 (A P0), the two sorted rows merged (count when oj == nullptr)
__global__ void prolong_merge_kernel(int64_t n, const int64_t* __restrict__ p0i, const int32_t* __restrict__ p0j,
                                     const double* __restrict__ p0a, const int64_t* __restrict__ qi, const int32_t* __restrict__ qj,
                                     const double* __restrict__ qa, const double* __restrict__ d, double omega, uint32_t* __restrict__ cnt,
                                     const uint32_t* __restrict__ off, int32_t* __restrict__ oj, double* __restrict__ oa) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double f = d[i] != 0.0 ? __ddiv_rn(omega, d[i]) : 0.0;
        int64_t p = p0i[i];
        const int64_t pe = p0i[i + 1];
        uint32_t k = 0;
        const int64_t o = oj ? (int64_t)off[i] : 0;
        for (int64_t q = qi[i]; q < qi[i + 1]; ++q) {
            const int32_t c = qj[q];
            for (; p < pe && p0j[p] < c; ++p, ++k)
                if (oj) { oj[o + k] = p0j[p]; oa[o + k] = p0a[p]; }
            double v = __dmul_rn(-f, qa[q]);
            if (p < pe && p0j[p] == c) { v = __dadd_rn(v, p0a[p]); ++p; }
            if (oj) { oj[o + k] = c; oa[o + k] = v; }
            ++k;
        }
        for (; p < pe; ++p, ++k)
            if (oj) { oj[o + k] = p0j[p]; oa[o + k] = p0a[p]; }
        if (cnt) cnt[i] = k;
    }
}

__global__ void u32_to_i64_kernel(int64_t n1, const uint32_t* __restrict__ a, int64_t* __restrict__ b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n1; i += (int64_t)gridDim.x * blockDim.x) b[i] = a[i];
}

// node of each dof (near null space levels: nodes are consecutive dof ranges)
__global__ void node_of_kernel(int64_t nn, const int64_t* __restrict__ node_ptr, int32_t* __restrict__ node_of) {
    for (int64_t I = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; I < nn; I += (int64_t)gridDim.x * blockDim.x)
        for (int64_t i = node_ptr[I]; i < node_ptr[I + 1]; ++i) node_of[i] = (int32_t)I;
}

// node graph of the dof graph (sp, sj): one warp per node, the nodes of its dofs' neighbours gathered in
// shared memory (cap entries per warp), sorted (bitonic), duplicates and the node itself removed; count
// (out == nullptr) or fill
constexpr int kCollapseMax = 16384;
__global__ void __launch_bounds__(128) collapse_kernel(int64_t nn, const int64_t* __restrict__ node_ptr, const uint32_t* __restrict__ sp,
                                                       const int32_t* __restrict__ sj, const int32_t* __restrict__ node_of, int cap,
                                                       uint32_t* __restrict__ cnt, const uint32_t* __restrict__ off,
                                                       int32_t* __restrict__ out, int* __restrict__ status) {
    extern __shared__ __align__(16) int32_t cbuf[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    int32_t* b = cbuf + (size_t)warp * cap;
    for (int64_t I = (int64_t)blockIdx.x * warps + warp; I < nn; I += (int64_t)gridDim.x * warps) {
        const uint32_t q0 = sp[node_ptr[I]], q1 = sp[node_ptr[I + 1]];
        const int len = (int)(q1 - q0);
        if (len > cap) {
            if (lane == 0) {
                atomicOr(status, kStOverflow);
                if (cnt) cnt[I] = 0;
            }
            continue;
        }
        int P = 1;
        while (P < len) P <<= 1;
        for (int k = lane; k < P; k += 32) {
            const int32_t J = k < len ? node_of[sj[q0 + k]] : INT32_MAX;
            b[k] = (J == (int32_t)I) ? INT32_MAX : J;
        }
        __syncwarp();
        for (int size = 2; size <= P; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int k = lane; k < P; k += 32) {
                    const int l = k ^ stride;
                    if (l > k) {
                        const bool up = (k & size) == 0;
                        const int32_t x = b[k], y = b[l];
                        if ((x > y) == up) { b[k] = y; b[l] = x; }
                    }
                }
                __syncwarp();
            }
        // distinct values: a position k counts when b[k] is real and differs from b[k - 1]
        uint32_t run = 0;
        for (int k0 = 0; k0 < P; k0 += 32) {
            const int k = k0 + lane;
            const bool keep = k < P && b[k] != INT32_MAX && (k == 0 || b[k] != b[k - 1]);
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (keep && out) out[off[I] + run + __popc(m & ((1u << lane) - 1u))] = b[k];
            run += __popc(m);
        }
        if (cnt && lane == 0) cnt[I] = run;
        __syncwarp();
    }
}

// longest gathered list of collapse_kernel: max over nodes of the node's dof rows' total length
__global__ void node_len_kernel(int64_t nn, const int64_t* __restrict__ node_ptr, const uint32_t* __restrict__ sp,
                                unsigned long long* __restrict__ out) {
    unsigned long long m = 0;
    for (int64_t I = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; I < nn; I += (int64_t)gridDim.x * blockDim.x)
        m = max(m, (unsigned long long)(sp[node_ptr[I + 1]] - sp[node_ptr[I]]));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// rigid body modes at the dof nodes: node coordinates from the first incident element's affine map
// (barycentric weights of the local node), then the six modes about the centroid c
__global__ void node_coords_kernel(int64_t nnodes, int n, const int64_t* __restrict__ inc_ptr, const int32_t* __restrict__ inc,
                                   const int32_t* __restrict__ tets, const double* __restrict__ xyz, const double* __restrict__ lam,
                                   double* __restrict__ out) {
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nnodes; m += (int64_t)gridDim.x * blockDim.x) {
        double x[3] = {0.0, 0.0, 0.0};
        if (inc_ptr[m + 1] > inc_ptr[m]) {
            const int32_t code = inc[inc_ptr[m]];
            const int64_t e = code >> 5;
            const int a = code & 31;
            for (int v = 0; v < 4; ++v) {
                const double w = lam[a * 4 + v];
                const int64_t g = tets[e * 4 + v];
                for (int d = 0; d < 3; ++d) x[d] = fma(w, xyz[g * 3 + d], x[d]);
            }
        }
        for (int d = 0; d < 3; ++d) out[m * 3 + d] = x[d];
    }
}
__global__ void rbm_kernel(int64_t nnodes, const double* __restrict__ xn, double cx, double cy, double cz, double* __restrict__ m0,
                           double* __restrict__ m1, double* __restrict__ m2, double* __restrict__ m3, double* __restrict__ m4,
                           double* __restrict__ m5) {
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nnodes; m += (int64_t)gridDim.x * blockDim.x) {
        const double x = xn[m * 3] - cx, y = xn[m * 3 + 1] - cy, z = xn[m * 3 + 2] - cz;
        const int64_t r = m * 3;
        m0[r] = 1.0; m0[r + 1] = 0.0; m0[r + 2] = 0.0;
        m1[r] = 0.0; m1[r + 1] = 1.0; m1[r + 2] = 0.0;
        m2[r] = 0.0; m2[r + 1] = 0.0; m2[r + 2] = 1.0;
        m3[r] = -y; m3[r + 1] = x; m3[r + 2] = 0.0;
        m4[r] = 0.0; m4[r + 1] = -z; m4[r + 2] = y;
        m5[r] = z; m5[r + 1] = 0.0; m5[r + 2] = -x;
    }
}

// Aggregation rounds (the host set-up's aggregate_mis2, amg_setup.cpp): states 0 undecided, 1 root,
// 2 out, 3 no strong neighbours; each kernel reads the previous step's arrays only.
__global__ void mis_init_kernel(int64_t n, const uint32_t* __restrict__ sp, int8_t* __restrict__ state) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        state[i] = sp[i + 1] > sp[i] ? 0 : 3;
}
// largest undecided key and any root in the closed neighbourhood (8 lanes per node, reductions by
// shuffles: max and or do not depend on the order). A neighbourhood without an undecided node (m1 = 0; no
// node's key is 0) is final and not looked at again: P2 48^3, 15 passes, 1530 -> 812 us.
constexpr int kMisLanes = 8;
__global__ void __launch_bounds__(256) mis_pass1_kernel(int64_t n, const uint32_t* __restrict__ sp, const int32_t* __restrict__ sj,
                                                        const int8_t* __restrict__ state, uint64_t* __restrict__ m1,
                                                        uint8_t* __restrict__ r1, bool first) {
    const int sub = threadIdx.x & (kMisLanes - 1);
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / kMisLanes);
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kMisLanes;; i += groups) {
        const bool live = i < n && (first || m1[i] != 0);
        uint64_t m = 0;
        unsigned r = 0;
        if (live) {
            if (sub == 0) {
                m = state[i] == 0 ? amg_mis_key(i) : 0;
                r = state[i] == 1;
            }
            for (uint32_t q = sp[i] + sub; q < sp[i + 1]; q += kMisLanes) {
                const int32_t j = sj[q];
                const int8_t sjs = state[j];
                if (sjs == 0) m = max(m, amg_mis_key(j));
                r |= sjs == 1;
            }
        }
        for (int o = kMisLanes / 2; o > 0; o >>= 1) {
            m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            r |= __shfl_xor_sync(0xffffffffu, r, o);
        }
        if (live && sub == 0) {
            m1[i] = m;
            r1[i] = (uint8_t)r;
        }
        // all lanes of the warp leave together (the shuffles above need them)
        if (__all_sync(0xffffffffu, i >= n)) break;
    }
}
// the same over distance 2, and the new state; counts the nodes left undecided
__global__ void __launch_bounds__(256) mis_pass2_kernel(int64_t n, const uint32_t* __restrict__ sp, const int32_t* __restrict__ sj,
                                                        const int8_t* __restrict__ state, const uint64_t* __restrict__ m1,
                                                        const uint8_t* __restrict__ r1, int8_t* __restrict__ nstate,
                                                        unsigned long long* __restrict__ undecided) {
    const int sub = threadIdx.x & (kMisLanes - 1);
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / kMisLanes);
    unsigned long long c = 0;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kMisLanes;; i += groups) {
        const bool live = i < n;
        const int8_t s0 = live ? state[i] : (int8_t)3;
        uint64_t m = 0;
        unsigned r = 0;
        if (live && s0 == 0) {
            if (sub == 0) {
                m = m1[i];
                r = r1[i];
            }
            for (uint32_t q = sp[i] + sub; q < sp[i + 1]; q += kMisLanes) {
                m = max(m, m1[sj[q]]);
                r |= r1[sj[q]];
            }
        }
        for (int o = kMisLanes / 2; o > 0; o >>= 1) {
            m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            r |= __shfl_xor_sync(0xffffffffu, r, o);
        }
        if (live && sub == 0) {
            int8_t ns = s0;
            if (s0 == 0) {
                if (r) ns = 2;
                else if (m == amg_mis_key(i)) ns = 1;
                else ++c;
            }
            nstate[i] = ns;
        }
        // all lanes of the warp leave together (the shuffles above need them)
        if (__all_sync(0xffffffffu, i >= n)) break;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(undecided, c);
}
__global__ void mis_root_flag_kernel(int64_t n, const int8_t* __restrict__ state, uint32_t* __restrict__ flag) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = state[i] == 1 ? 1u : 0u;
}
// roots and their neighbours (a node has at most one root neighbour)
__global__ void mis_assign1_kernel(int64_t n, const uint32_t* __restrict__ sp, const int32_t* __restrict__ sj,
                                   const int8_t* __restrict__ state, const uint32_t* __restrict__ rank, int32_t* __restrict__ a1) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t a = -1;
        if (state[i] == 1) {
            a = (int32_t)rank[i];
        } else {
            for (uint32_t q = sp[i]; q < sp[i + 1]; ++q)
                if (state[sj[q]] == 1) { a = (int32_t)rank[sj[q]]; break; }
        }
        a1[i] = a;
    }
}
// the other coupled nodes join the aggregate of their first neighbour (column order) aggregated above
__global__ void mis_assign2_kernel(int64_t n, const uint32_t* __restrict__ sp, const int32_t* __restrict__ sj,
                                   const int8_t* __restrict__ state, const int32_t* __restrict__ a1, int32_t* __restrict__ agg) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t a = a1[i];
        if (a < 0 && state[i] != 3)
            for (uint32_t q = sp[i]; q < sp[i + 1]; ++q)
                if (a1[sj[q]] >= 0) { a = a1[sj[q]]; break; }
        agg[i] = a;
    }
}
// tentative scaling of the constant vector: aggregate sizes, then 1/sqrt(size)
__global__ void agg_size_kernel(int64_t n, const int32_t* __restrict__ agg, unsigned int* __restrict__ sz) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (agg[i] >= 0) atomicAdd(sz + agg[i], 1u);
}
__global__ void agg_scale_kernel(int64_t nagg, const unsigned int* __restrict__ sz, double* __restrict__ s0) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < nagg; c += (int64_t)gridDim.x * blockDim.x)
        s0[c] = __ddiv_rn(1.0, __dsqrt_rn((double)sz[c]));
}

// Sparse product C = A B, G lanes per row of A. The lanes take one entry of A's row after another and
// beside it G products with the entry's row of B, whose columns are distinct: no two lanes of a step meet
// in an output entry, and every output entry is its products' sum in the order of A's row, the host's.
// Each group has a hash table of T slots in shared memory (slot h of group g at h * (32 / G) + g). kCount:
// cnt[i] = distinct columns of row i, or row i appended to `ovf` when it holds more than `cap` (status
// overflow when ovf is null). kFill: rows whose count exceeds the cap are left to a larger table; the others
// are written sorted at off[i]. kPadded: both at once, the row written sorted at i * cap, from where
// pad_copy_kernel takes it to its place once the counts are summed. The groups of a warp run in step (each on its own entry),
// a step's columns and values loaded during the step before it, the entries of A's row two groups ahead.
// Bound: the FP64 pipe (a warp's product and sum occupy it 32 cycles) and instruction issue, each busy two
// thirds of the time. P2 48^3, A P (25.8 M entries x 4): 1150 us to count and 2910 to fill -> 1710 padded
// and 70 to copy; R (A P): 461 + 728 -> 603 + 7, against one warp per row that numbered 32 products at a
// time by a search over the row's prefix sums and grouped equal columns by __match_any_sync. Four lanes a row
// give 1600 on A P and lose a third on the next level; two 1600-2300, one 2700-5100.
struct SpgemmArgs {
    int64_t nrows = 0;
    const int32_t* rows = nullptr;   // row list (null: rows 0..nrows-1)
    const int64_t* ia = nullptr;
    const int32_t* ja = nullptr;
    const double* a = nullptr;
    const int64_t* ib = nullptr;
    const int32_t* jb = nullptr;
    const double* b = nullptr;
    int tsize = 256;                 // hash slots per row (power of two, >= 64)
    int tshift = 24;                 // 32 - log2(tsize)
    int warps = 8;                   // warps per block
    int wbytes = 0;                  // shared memory per warp
    uint32_t* cnt = nullptr;
    int32_t* ovf = nullptr;
    uint32_t* novf = nullptr;
    const int64_t* off = nullptr;
    int32_t* oj = nullptr;
    double* oa = nullptr;
    int* status = nullptr;
};

constexpr int kRankMax = 128;        // rows up to this long are sorted by counting smaller columns
// The longest row that a table keeps; longer ones are listed for the next. Only a whole warp can sort more than
// kRankMax columns (the bitonic sort).
__host__ __device__ constexpr int spgemm_cap(int tsize, int group) {
    const int c = group <= 8 ? tsize - tsize / 4 : tsize / 2;
    return group == 32 || c <= kRankMax ? c : kRankMax;
}
int spgemm_warp_bytes(int tsize, int group, bool fill) {
    return tsize * (32 / group) * ((fill ? 8 : 0) + 4 + 2);
}

enum { kCount, kFill, kPadded };

template <int G, int MODE>
__global__ void __launch_bounds__(256) spgemm_kernel(SpgemmArgs g) {
    extern __shared__ __align__(16) unsigned char sg_smem[];
    constexpr int NG = 32 / G;
    constexpr bool FILL = MODE != kCount;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & (G - 1), grp = lane / G;
    const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (grp * G);
    static_assert(G == 32 || spgemm_cap(kBins[kNumBins - 1], G) <= kRankMax, "a row that is counted has to be written");
    const int T = g.tsize, cap = spgemm_cap(T, G);
    unsigned char* base = sg_smem + (size_t)warp * g.wbytes;
    double* hv = reinterpret_cast<double*>(base) + grp;                                        // values
    int32_t* hk = reinterpret_cast<int32_t*>(base + (FILL ? (size_t)T * NG * 8 : 0)) + grp;    // keys (-1: empty)
    uint16_t* list = reinterpret_cast<uint16_t*>(hk - grp + T * NG) + grp;                     // used slots
    for (int k = sub; k < T; k += G) hk[k * NG] = -1;
    __syncwarp();
    const int64_t step = (int64_t)gridDim.x * g.warps * NG;
    for (int64_t r0 = ((int64_t)blockIdx.x * g.warps + warp) * NG; r0 < g.nrows; r0 += step) {
        const int64_t r = r0 + grp;
        bool act = r < g.nrows;
        int64_t i = 0, ob = 0;
        uint32_t a0 = 0;
        int na = 0;
        if (act) {
            i = g.rows ? (int64_t)g.rows[r] : r;
            if (MODE == kFill) {
                ob = g.off[i];
                act = g.off[i + 1] - ob <= cap;                     // else a larger table's row
            }
            if (MODE == kPadded) ob = i * cap;
            a0 = (uint32_t)g.ia[i];                                  // all factors have fewer than 2^32 entries
            na = act ? (int)((uint32_t)g.ia[i + 1] - a0) : 0;
        }
        const bool mine = act;
        int nuniq = 0;
        bool over = false;
        // the group's place: entry e of the row, product q of the entry; lane `sub` holds the entries
        // congruent to it of the current G
        int e = -1, q = 0, len = 0;
        uint32_t bstart = 0, cb = 0;
        int clen = 0;
        double av = 0.0, ca = 0.0;
        int32_t ncol = -1;
        double nb_ = 0.0, na_ = 0.0;
        // entries t .. t + G - 1 (their columns loaded before), and the columns of the G after them
        uint32_t pb = 0, pe = 0;
        int32_t pc = 0;
        double pa = 0.0;
        auto ahead = [&](int t) {
            if (t + sub < na) {
                pb = (uint32_t)g.ib[pc];
                pe = (uint32_t)g.ib[pc + 1];
                if (FILL) pa = g.a[a0 + t + sub];
            }
            if (t + G + sub < na) pc = g.ja[a0 + t + G + sub];
        };
        if (sub < na) pc = g.ja[a0 + sub];
        ahead(0);
        auto advance = [&]() {                                       // the next step's column and value
            const bool next = e < na && q + G >= len;
            if (next) {
                ++e;
                q = 0;
            } else {
                q += G;
            }
            if (next && e < na && (e & (G - 1)) == 0) {              // the next G entries; those after them on their way
                cb = pb;
                clen = (int)(pe - pb);
                ca = pa;
                ahead(e + G);
            }
            const int src = (e & (G - 1)) + grp * G;
            const uint32_t sb = __shfl_sync(0xffffffffu, cb, src);
            const int sl = __shfl_sync(0xffffffffu, clen, src);
            if (FILL) av = __shfl_sync(0xffffffffu, ca, src);
            if (next) {
                bstart = sb;
                len = sl;
            }
            ncol = -1;
            if (e < na && q + sub < len) {
                ncol = g.jb[bstart + q + sub];
                if (FILL) {
                    nb_ = g.b[bstart + q + sub];
                    na_ = av;
                }
            }
        };
        advance();
        while (__any_sync(0xffffffffu, e < na)) {
            const int32_t col = ncol;
            const double va = na_, vb = nb_;
            advance();
            int slot = -1;
            bool newkey = false;
            if (col >= 0) {
                uint32_t h = ((uint32_t)col * 2654435761u) >> g.tshift;
                for (int probe = 0; probe < T; ++probe) {
                    int32_t old = hk[h * NG];
                    if (old == -1) old = atomicCAS(hk + h * NG, -1, col);
                    if (old == -1) { newkey = true; slot = (int)h; break; }
                    if (old == col) { slot = (int)h; break; }
                    h = (h + 1) & (uint32_t)(T - 1);
                }
            }
            const unsigned nb = __ballot_sync(0xffffffffu, newkey) & gmask;
            if (newkey) {
                const int pos = nuniq + __popc(nb & ((1u << lane) - 1u));
                if (pos < cap) list[pos * NG] = (uint16_t)slot;
            }
            nuniq += __popc(nb);
            if (FILL && slot >= 0) hv[slot * NG] = __dadd_rn(newkey ? 0.0 : hv[slot * NG], __dmul_rn(va, vb));
            if (nuniq > cap && !over) {                             // the row ends here: at most cap + G slots used
                over = true;
                na = e = 0;
                ncol = -1;
            }
            __syncwarp();
        }
        if (over) {
            for (int k = sub; k < T; k += G) hk[k * NG] = -1;
            if (sub == 0) {
                if (MODE != kFill && g.ovf) g.ovf[atomicAdd(g.novf, 1u)] = (int32_t)i;
                else atomicOr(g.status, kStOverflow);
                if (MODE != kFill) g.cnt[i] = 0;
            }
            nuniq = 0;
        } else if (MODE != kFill && mine && sub == 0) {
            g.cnt[i] = (uint32_t)nuniq;
        }
        if (FILL && nuniq <= kRankMax) {
            // place of a column: the number of smaller ones in the row
            for (int k = sub; k < nuniq; k += G) {
                const int s = list[k * NG];
                const int32_t key = hk[s * NG];
                int rank = 0;
                for (int m = 0; m < nuniq; ++m) rank += hk[list[m * NG] * NG] < key;
                g.oj[ob + rank] = key;
                g.oa[ob + rank] = hv[s * NG];
            }
        } else if (FILL && G == 32) {        // (narrower groups keep no row above kRankMax)
            // bitonic sort of the used slots by key (padding last), then the row
            int P = 1;
            while (P < nuniq) P <<= 1;
            constexpr uint16_t kPad = 0xffff;
            for (int k = nuniq + lane; k < P; k += 32) list[k] = kPad;
            __syncwarp();
            for (int size = 2; size <= P; size <<= 1)
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    for (int k = lane; k < P; k += 32) {
                        const int l = k ^ stride;
                        if (l > k) {
                            const bool up = (k & size) == 0;
                            const uint16_t sa = list[k], sb = list[l];
                            const int32_t ka = sa == kPad ? INT32_MAX : hk[sa], kb = sb == kPad ? INT32_MAX : hk[sb];
                            if ((ka > kb) == up) {
                                list[k] = sb;
                                list[l] = sa;
                            }
                        }
                    }
                    __syncwarp();
                }
            for (int k = lane; k < nuniq; k += 32) {
                const int s = list[k];
                g.oj[ob + k] = hk[s];
                g.oa[ob + k] = hv[s];
            }
        }
        __syncwarp();
        for (int k = sub; k < nuniq; k += G) hk[list[k * NG] * NG] = -1;
        __syncwarp();
    }
}

// A P0 for the tentative prolongator of the constant vector (row j of P0: s0[agg_j] at column agg_j, or
// empty): one thread per row with a table of its own, T columns in first-met order, searched from the last
// hit on; the row's products summed in its order. Modes as above; rows
// with more than T columns go to the general product. P2 48^3: 793 us to count and 1740 to fill -> 433
// padded and 50 to copy (FP64 pipe half busy, table latency).
constexpr int kAp0T = 16;
template <int MODE>
__global__ void __launch_bounds__(128) ap0_kernel(SpgemmArgs g, const int32_t* __restrict__ agg, const double* __restrict__ s0) {
    constexpr bool FILL = MODE != kCount;
    __shared__ int32_t tk[kAp0T][128];
    __shared__ double tv[FILL ? kAp0T : 1][128];
    const int t = threadIdx.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + t; i < g.nrows; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t ob = 0;
        if (MODE == kFill) {
            ob = g.off[i];
            if (g.off[i + 1] - ob > kAp0T) continue;
        }
        if (MODE == kPadded) ob = i * kAp0T;
        const int64_t pe = g.ia[i + 1];
        int n = 0, last = 0;
        bool over = false;
        for (int64_t p = g.ia[i]; p < pe && !over; p += 4) {
            int32_t c[4];
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = p + u < pe ? g.ja[p + u] : -1;
                if (FILL) v[u] = p + u < pe ? g.a[p + u] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] = c[u] >= 0 ? agg[c[u]] : -1;
            if (FILL) {
                double w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) w[u] = c[u] >= 0 ? s0[c[u]] : 0.0;
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = __dmul_rn(v[u], w[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (c[u] < 0) continue;
                if (n == 0 || tk[last][t] != c[u]) {
                    int k = 0;
                    while (k < n && tk[k][t] != c[u]) ++k;
                    if (k == n) {
                        if (n == kAp0T) { over = true; break; }
                        tk[n][t] = c[u];
                        if (FILL) tv[n][t] = 0.0;
                        ++n;
                    }
                    last = k;
                }
                if (FILL) tv[last][t] = __dadd_rn(tv[last][t], v[u]);
            }
        }
        if (MODE != kFill) {
            if (over) g.ovf[atomicAdd(g.novf, 1u)] = (int32_t)i;
            g.cnt[i] = over ? 0u : (uint32_t)n;
        }
        if (FILL && !over) {
            for (int k = 0; k < n; ++k) {
                const int32_t key = tk[k][t];
                int rank = 0;
                for (int m = 0; m < n; ++m) rank += tk[m][t] < key;
                g.oj[ob + rank] = key;
                g.oa[ob + rank] = tv[k][t];
            }
        }
    }
}

// rows written padded (row i at i * pad) to their places; longer rows are written there by their own pass
__global__ void __launch_bounds__(256) pad_copy_kernel(int64_t n, int pad, const int64_t* __restrict__ off,
                                                       const int32_t* __restrict__ pj, const double* __restrict__ pa,
                                                       int32_t* __restrict__ oj, double* __restrict__ oa) {
    const int sub = threadIdx.x & 7;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3; i < n; i += ((int64_t)gridDim.x * blockDim.x) >> 3) {
        const int64_t o = off[i];
        const int len = (int)(off[i + 1] - o);
        if (len > pad) continue;
        for (int k = sub; k < len; k += 8) {
            oj[o + k] = pj[i * pad + k];
            oa[o + k] = pa[i * pad + k];
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------------------------------

struct SpgemmTable { int group, tsize, log2; };

template <int G, int MODE>
int launch_spgemm_g(fgpu_ctx* ctx, SpgemmArgs g, const SpgemmTable& t) {
    g.tsize = t.tsize;
    g.tshift = 32 - t.log2;
    g.wbytes = spgemm_warp_bytes(t.tsize, G, MODE != kCount);
    const int rows = 32 / G;
    // few rows: one warp a block, so that they spread over the SMs
    const int spread = (int)std::max<int64_t>(1, g.nrows / (152 * rows));
    g.warps = std::max(1, std::min({8, spread, (110 * 1024) / g.wbytes}));
    const int smem = g.warps * g.wbytes;
    auto kernel = spgemm_kernel<G, MODE>;
    DEV_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int per_sm = std::max(1, std::min(2048 / (32 * g.warps), (228 * 1024) / (smem + 1024)));
    const int blocks = grid_rows(g.nrows, g.warps * rows, 152 * per_sm);
    kernel<<<blocks, 32 * g.warps, smem, ctx->stream>>>(g);
    ctx->launches++;
    DEV_TRY(cudaGetLastError());
    return FGPU_OK;
}
template <int MODE>
int launch_spgemm(fgpu_ctx* ctx, const SpgemmArgs& g, const SpgemmTable& t) {
    if (t.group == 8) return launch_spgemm_g<8, MODE>(ctx, g, t);
    if (t.group == 16) return launch_spgemm_g<16, MODE>(ctx, g, t);
    return launch_spgemm_g<32, MODE>(ctx, g, t);
}

// C = A B (rows sorted by column). agg, s0: B is the tentative prolongator of the constant vector.
// *overflow: a row with more distinct columns than the largest table.
// Table and lanes per row: the first pass takes 8 lanes up to a mean of 8 entries in B's rows, else 16 (a
// step of 16 lanes on rows of 13 entries does as much as two of 8), with 256 slots where a row has many
// products and 64 else; a level of few rows takes whole warps, its time one row's chain of steps. Rows that
// do not fit go on to whole warps with the next larger table. Neither line is sharp (prolongation and Galerkin
// products of a set-up, ms): 64 slots up to 512 products a row P2 48^3 5.3, P1 64^3 1.9, rigid body modes P2 16^3
// 20.4, the same from 200 to 800; never 7.0 / 2.1 / 20.4, up to 2000 5.3 / 2.2 / 22.0. Groups from 4096 rows P2 48^3
// 5.3, P3 24^3 4.7, from 1024 5.3 / 4.8, 8192 5.3 / 4.7, 16384 5.4 / 4.7, always whole warps 10.4 / 6.6.
int spgemm_once(fgpu_ctx* ctx, const AmgDevCsr& A, const AmgDevCsr& B, AmgDevCsr& C, int* d_status, bool* overflow,
                const int32_t* agg, const double* s0, bool* padded_form) {
    *overflow = false;
    const int64_t n = A.nrows;
    SpgemmTable first = {32, 256, 8};
    const double ma = (double)A.nnz / std::max<int64_t>(A.nrows, 1), mb = (double)B.nnz / std::max<int64_t>(B.nrows, 1);
    if (n >= kGroupRows && mb <= 24.0) {
        first.group = mb <= 8.0 ? 8 : 16;
        if (ma * mb <= 512.0) first = {first.group, 64, 6};
    }
    SpgemmTable tables[1 + kNumBins];
    int nt = 0;
    tables[nt++] = first;
    for (int k = 0; k < kNumBins; ++k)
        if (kBins[k] > first.tsize) tables[nt++] = {32, kBins[k], kBinLog[k]};
    if (agg) {                                   // then the first table is ap0_kernel's own
        tables[0] = {1, kAp0T, 0};
        nt = 1;
        for (int k = 0; k < kNumBins; ++k) tables[nt++] = {32, kBins[k], kBinLog[k]};
    }
    Work w(ctx);
    uint32_t* cnt = w.get<uint32_t>(n + 1);
    uint32_t* off32 = w.get<uint32_t>(n + 1);
    uint32_t* novf = w.get<uint32_t>(1 + kNumBins);
    int32_t* ovf[1 + kNumBins] = {nullptr};
    DEV_ALLOC(cnt && off32 && novf);
    DEV_TRY(cudaMemsetAsync(novf, 0, (1 + kNumBins) * sizeof(uint32_t), ctx->stream));
    SpgemmArgs g;
    g.ia = A.ia; g.ja = A.ja; g.a = A.a;
    g.ib = B.ia; g.jb = B.ja; g.b = B.a;
    g.status = d_status;
    auto launch = [&](SpgemmArgs& x, int k, int mode) -> int {
        if (!agg || k > 0)
            return mode == kCount ? launch_spgemm<kCount>(ctx, x, tables[k])
                                  : mode == kFill ? launch_spgemm<kFill>(ctx, x, tables[k]) : launch_spgemm<kPadded>(ctx, x, tables[k]);
        const int blocks = grid_rows(n, 128);
        if (mode == kCount) ap0_kernel<kCount><<<blocks, 128, 0, ctx->stream>>>(x, agg, s0);
        else if (mode == kFill) ap0_kernel<kFill><<<blocks, 128, 0, ctx->stream>>>(x, agg, s0);
        else ap0_kernel<kPadded><<<blocks, 128, 0, ctx->stream>>>(x, agg, s0);
        ctx->launches++;
        DEV_TRY(cudaGetLastError());
        return FGPU_OK;
    };
    // the first table's rows in one pass where their padded form stays small (2 GB, 3.7 M rows, and four
    // entries to one of A), which saves the count pass (P2 48^3: 1.8 of 20 ms of set-up)
    const int pad = agg ? kAp0T : spgemm_cap(first.tsize, first.group);
    int32_t* pj = nullptr;
    double* pa = nullptr;
    *padded_form = *padded_form && n * pad * 12 <= kPadBytes && n * pad <= 4 * A.nnz;
    if (*padded_form) {
        pj = w.get<int32_t>(n * pad);
        pa = pj ? w.get<double>(n * pad) : nullptr;
        if (!pa) pj = nullptr;                   // no room: counted first
    }
    // count: all rows with the first table, the rows it cannot hold with the next ones in turn
    int64_t rows_in[1 + kNumBins] = {n};
    for (int k = 0; k < nt && rows_in[k] > 0; ++k) {
        SpgemmArgs c = g;
        c.nrows = rows_in[k];
        c.rows = ovf[k];
        c.cnt = cnt;
        if (k + 1 < nt) {
            DEV_ALLOC(ovf[k + 1] = w.get<int32_t>(rows_in[k]));
            c.ovf = ovf[k + 1];
            c.novf = novf + k + 1;
        }
        const bool padded = k == 0 && pj;
        if (padded) { c.oj = pj; c.oa = pa; }
        int rc = launch(c, k, padded ? kPadded : kCount);
        if (rc) return rc;
        if (k + 1 < nt) {
            uint32_t hn = 0;
            DEV_TRY(cudaMemcpyAsync(&hn, novf + k + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
            DEV_TRY(cudaStreamSynchronize(ctx->stream));
            rows_in[k + 1] = hn;
        }
    }
    int st = 0;
    int rc = read_status(ctx, d_status, &st);
    if (rc) return rc;
    if (st & kStOverflow) { *overflow = true; return FGPU_OK; }
    uint64_t total = 0;
    rc = scan_u32(ctx, cnt, off32, n, &total);
    if (rc) return rc;
    rc = alloc_csr(ctx, C, n, B.ncols, (int64_t)total);
    if (rc) return rc;
    u32_to_i64_kernel<<<grid_rows(n + 1, 256), 256, 0, ctx->stream>>>(n + 1, off32, C.ia);
    ctx->launches++;
    g.off = C.ia; g.oj = C.ja; g.oa = C.a;
    if (pj) {
        pad_copy_kernel<<<grid_rows(n, 32), 256, 0, ctx->stream>>>(n, pad, C.ia, pj, pa, C.ja, C.a);
        ctx->launches++;
    }
    for (int k = pj ? 1 : 0; k < nt && rows_in[k] > 0; ++k) {
        SpgemmArgs f = g;
        f.nrows = rows_in[k];
        f.rows = ovf[k];
        rc = launch(f, k, kFill);
        if (rc) return rc;
    }
    rc = read_status(ctx, d_status, &st);
    if (rc) return rc;
    *overflow = (st & kStOverflow) != 0;
    return FGPU_OK;
}
// Where the padded form leaves no room for the product itself, the rows are counted first.
int spgemm_dev(fgpu_ctx* ctx, const AmgDevCsr& A, const AmgDevCsr& B, AmgDevCsr& C, int* d_status, bool* overflow,
               const int32_t* agg = nullptr, const double* s0 = nullptr) {
    bool padded = true;
    const int rc = spgemm_once(ctx, A, B, C, d_status, overflow, agg, s0, &padded);
    if (!padded || (rc != FGPU_ERR_ALLOC && !(rc == FGPU_ERR_CUDA && cudaPeekAtLastError() == cudaErrorMemoryAllocation))) return rc;
    cudaGetLastError();
    padded = false;
    return spgemm_once(ctx, A, B, C, d_status, overflow, agg, s0, &padded);
}

int seg_sort(fgpu_ctx* ctx, int64_t n, const uint32_t* off32, const int64_t* off64, int32_t* key, double* val, int* d_status) {
    unsigned long long* dmax = nullptr;
    DEV_TRY(pool_malloc(ctx->stream, &dmax, sizeof(unsigned long long)));
    struct Free { unsigned long long* p; ~Free() { pool_free(p); } } fr{dmax};
    DEV_TRY(cudaMemsetAsync(dmax, 0, sizeof(unsigned long long), ctx->stream));
    max_row_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, off32, off64, dmax);
    unsigned long long hmax = 0;
    DEV_TRY(cudaMemcpyAsync(&hmax, dmax, sizeof(hmax), cudaMemcpyDeviceToHost, ctx->stream));
    DEV_TRY(cudaStreamSynchronize(ctx->stream));
    ctx->launches++;
    if (hmax <= 1) return FGPU_OK;
    int cap = 32;
    while (cap < (int)std::min<unsigned long long>(hmax, (unsigned long long)kSortMax + 1)) cap <<= 1;
    cap = std::min(cap, kSortMax);              // longer rows raise the overflow status
    const int bytes = val ? 12 : 4;
    const int warps = std::max(1, std::min(4, (96 * 1024) / (cap * bytes)));
    const int smem = warps * cap * bytes;
    DEV_TRY(cudaFuncSetAttribute(seg_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    seg_sort_kernel<<<grid_rows(n, warps, 152 * 8), warps * 32, smem, ctx->stream>>>(n, off32, off64, cap, key, val, d_status);
    ctx->launches++;
    DEV_TRY(cudaGetLastError());
    return FGPU_OK;
}

// T = M^T of an n x m device CSR (rows of T sorted by column of M)
int transpose_dev(fgpu_ctx* ctx, const AmgDevCsr& M, AmgDevCsr& T, int* d_status) {
    const int64_t m = M.ncols;
    Work w(ctx);
    uint32_t* tcnt = w.get<uint32_t>(m + 1);
    uint32_t* toff = w.get<uint32_t>(m + 1);
    uint32_t* cur = w.get<uint32_t>(m + 1);
    DEV_ALLOC(tcnt && toff && cur);
    DEV_TRY(cudaMemsetAsync(tcnt, 0, (m + 1) * sizeof(uint32_t), ctx->stream));
    col_count_kernel<<<grid_rows(M.nnz, 256), 256, 0, ctx->stream>>>(M.nnz, M.ja, tcnt);
    ctx->launches++;
    int rc = scan_u32(ctx, tcnt, toff, m, nullptr);
    if (rc) return rc;
    rc = alloc_csr(ctx, T, m, M.nrows, M.nnz);
    if (rc) return rc;
    DEV_TRY(cudaMemcpyAsync(cur, toff, (m + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
    transpose_fill_kernel<<<grid_rows(M.nrows, 256), 256, 0, ctx->stream>>>(M.nrows, nullptr, M.ia, M.ja, M.a, cur, T.ja, T.a);
    u32_to_i64_kernel<<<grid_rows(m + 1, 256), 256, 0, ctx->stream>>>(m + 1, toff, T.ia);
    ctx->launches += 2;
    rc = seg_sort(ctx, m, nullptr, T.ia, T.ja, T.a, d_status);
    if (rc) return rc;
    DEV_TRY(cudaStreamSynchronize(ctx->stream));     // the scratch above is freed on return
    return FGPU_OK;
}

// lambda_max(D^-1 A) by Lanczos on its own stream, driven by its own host thread (it runs beside the
// aggregation and the first products); the same arithmetic as the host set-up's estimate
struct LanczosJob {
    int64_t n = 0;
    const int64_t* ia = nullptr;
    const int32_t* ja = nullptr;
    const double* a = nullptr;
    const double* d = nullptr;
    double *s = nullptr, *v = nullptr, *vold = nullptr, *wv = nullptr, *u = nullptr, *part = nullptr;
    LanczosScalars* sc = nullptr;
    int32_t *perm = nullptr, *slice_len = nullptr;
    cudaStream_t st = nullptr;
    double lmax = 0;
    int launches = 0;
    cudaError_t err = cudaSuccess;

    bool ok(cudaError_t e) {
        if (e != cudaSuccess && err == cudaSuccess) err = e;
        return e == cudaSuccess;
    }
    int device = 0;
    void run() {
        if (!ok(cudaSetDevice(device))) return;
        sell_order_launch(st, n, ia, perm, slice_len);
        const int nch = (int)((n + kLanczosChunk - 1) / kLanczosChunk);
        const int g = grid_rows(n, 256);
        if (!ok(cudaMemsetAsync(sc, 0, sizeof(LanczosScalars), st))) return;
        lanczos_random_kernel<<<nch, 128, 0, st>>>(n, v, part, sc);
        lanczos_start_kernel<<<g, 256, 0, st>>>(n, d, s, v, vold, u, sc);
        launches += 3;
        for (int k = 0; k < kLanczosSteps; ++k) {
            lanczos_spmv_kernel<<<grid_rows(n, 64), 256, 0, st>>>(n, ia, ja, a, perm, s, u, wv, sc);
            lanczos_dot_kernel<false><<<nch, 128, 0, st>>>(n, k, v, vold, wv, part, sc);
            lanczos_dot_kernel<true><<<nch, 128, 0, st>>>(n, k, v, vold, wv, part, sc);
            launches += 3;
            if (k + 1 < kLanczosSteps) {
                lanczos_next_kernel<<<g, 256, 0, st>>>(n, k, s, wv, v, vold, u, sc);
                ++launches;
            }
        }
        LanczosScalars h;
        if (!ok(cudaGetLastError()) || !ok(cudaMemcpyAsync(&h, sc, sizeof(h), cudaMemcpyDeviceToHost, st)) || !ok(cudaStreamSynchronize(st)))
            return;
        lmax = amg_tridiag_lmax(std::vector<double>(h.al, h.al + h.steps), std::vector<double>(h.be, h.be + h.steps - 1));
    }
};

// One level on the device: lambda_max, strength graph, aggregation, P, R, A_c = R (A P).
// *handoff: the level goes to the host set-up instead (a row beyond a kernel's capacity, or nothing
// to coarsen); *last: the coarsening stagnates and A_c is the coarsest operator.
int level_dev(fgpu_ctx* ctx, AmgDevLevel& L, const AmgHostCfg& cfg, const AmgNns* nns, AmgNns* next, int* d_status, AmgDevCsr& Ac,
              bool* handoff, bool* last, AmgSetupTimes& tm) {
    using clock = std::chrono::steady_clock;
    auto ms_since = [](clock::time_point t) { return std::chrono::duration<double, std::milli>(clock::now() - t).count(); };
    auto tphase = clock::now();
    *handoff = false;
    *last = false;
    const AmgDevCsr& A = L.A;
    const int64_t n = A.nrows;
    const int64_t nch = (n + kLanczosChunk - 1) / kLanczosChunk;
    Work w(ctx);
    double* d = w.get<double>(n);
    uint32_t* cnt = w.get<uint32_t>(n + 1);
    uint32_t* tp = w.get<uint32_t>(n + 1);
    LanczosJob lz;
    lz.n = n; lz.ia = A.ia; lz.ja = A.ja; lz.a = A.a; lz.d = d; lz.device = ctx->device;
    lz.s = w.get<double>(n);
    lz.v = w.get<double>(n);
    lz.vold = w.get<double>(n);
    lz.wv = w.get<double>(n);
    lz.u = w.get<double>(n);
    lz.part = w.get<double>(nch);
    lz.sc = w.get<LanczosScalars>(1);
    lz.perm = w.get<int32_t>(n);
    lz.slice_len = w.get<int32_t>((n + 31) / 32);
    DEV_ALLOC(d && cnt && tp && lz.s && lz.v && lz.vold && lz.wv && lz.u && lz.part && lz.sc && lz.perm && lz.slice_len);
    diag_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, A.ia, A.ja, A.a, d, d_status);
    ctx->launches++;
    // the Lanczos thread and stream: started once the diagonal is formed, joined before any return
    std::thread lanczos;
    cudaEvent_t d_ready = nullptr;
    struct LanczosGuard {
        std::thread& t;
        LanczosJob& job;
        cudaEvent_t& ev;
        ~LanczosGuard() {
            if (t.joinable()) t.join();
            if (job.st) {
                cudaStreamSynchronize(job.st);     // the job's arrays go back to the pool of another stream
                cudaStreamDestroy(job.st);
            }
            if (ev) cudaEventDestroy(ev);
        }
    } lanczos_guard{lanczos, lz, d_ready};
    DEV_TRY(cudaEventCreateWithFlags(&d_ready, cudaEventDisableTiming));
    DEV_TRY(cudaEventRecord(d_ready, ctx->stream));
    DEV_TRY(cudaStreamCreateWithFlags(&lz.st, cudaStreamNonBlocking));
    DEV_TRY(cudaStreamWaitEvent(lz.st, d_ready, 0));
    lanczos = std::thread([&lz] { lz.run(); });
    strong_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, A.ia, A.ja, A.a, d, cfg.threshold, cnt, nullptr, nullptr);
    ctx->launches++;
    uint64_t ns = 0;
    int rc = scan_u32(ctx, cnt, tp, n, &ns);
    if (rc) return rc;
    int st = 0;
    rc = read_status(ctx, d_status, &st);
    if (rc) return rc;
    if (st & kStDiag) { ctx->err = "gamg: the diagonal must be positive (SPD matrix)"; return FGPU_ERR_INVALID; }
    // strength graph S, its rows in column order
    int32_t* tmpj = w.get<int32_t>((int64_t)ns);
    DEV_ALLOC(tmpj);
    strong_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, A.ia, A.ja, A.a, d, cfg.threshold, nullptr, tp, tmpj);
    ctx->launches++;
    // the graph to aggregate: the symmetrised dof graph S + S^T, or (near null space) its node graph,
    // formed as N(S) + N(S)^T (the same sorted rows as N(S + S^T): a node pair is coupled when any of
    // their dofs are, in either direction), which symmetrises the node graph instead of the nine-times
    // larger dof graph of a 3-component operator (vector P2 48^3 beam, the set-up run alone: graph phase
    // 113 -> 54 ms, set-up 750 -> 705 ms, the Lanczos estimate on its own stream now overlapping the
    // aggregation; after the other solves of the elasticity workload 742 ms)
    int64_t ng = n;
    const uint32_t* gp = tp;
    const int32_t* gjs = tmpj;
    if (nns) {
        ng = (int64_t)nns->node_ptr.size() - 1;
        int64_t* dnp = w.get<int64_t>(ng + 1);
        int32_t* node_of = w.get<int32_t>(n);
        uint32_t* ncnt = w.get<uint32_t>(ng + 1);
        uint32_t* np32 = w.get<uint32_t>(ng + 1);
        DEV_ALLOC(dnp && node_of && ncnt && np32);
        unsigned long long* dmax = w.get<unsigned long long>(1);
        DEV_ALLOC(dmax);
        DEV_TRY(cudaMemcpyAsync(dnp, nns->node_ptr.data(), (ng + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
        DEV_TRY(cudaMemsetAsync(dmax, 0, sizeof(unsigned long long), ctx->stream));
        node_of_kernel<<<grid_rows(ng, 256), 256, 0, ctx->stream>>>(ng, dnp, node_of);
        node_len_kernel<<<grid_rows(ng, 256), 256, 0, ctx->stream>>>(ng, dnp, tp, dmax);
        unsigned long long hmax = 0;
        DEV_TRY(cudaMemcpyAsync(&hmax, dmax, sizeof(hmax), cudaMemcpyDeviceToHost, ctx->stream));
        DEV_TRY(cudaStreamSynchronize(ctx->stream));
        if (hmax > (unsigned long long)kCollapseMax) { *handoff = true; tm.handoff = 2; return FGPU_OK; }
        int cap = 32;
        while (cap < (int)hmax) cap <<= 1;
        const int cwarps = std::max(1, std::min(4, (96 * 1024) / (cap * 4)));
        const int csmem = cwarps * cap * 4;
        DEV_TRY(cudaFuncSetAttribute(collapse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, csmem));
        collapse_kernel<<<grid_rows(ng, cwarps, 152 * 8), cwarps * 32, csmem, ctx->stream>>>(ng, dnp, tp, tmpj, node_of, cap, ncnt, nullptr,
                                                                                            nullptr, d_status);
        ctx->launches += 3;
        uint64_t nnj = 0;
        rc = scan_u32(ctx, ncnt, np32, ng, &nnj);
        if (rc) return rc;
        int32_t* nj = w.get<int32_t>((int64_t)nnj);
        DEV_ALLOC(nj);
        collapse_kernel<<<grid_rows(ng, cwarps, 152 * 8), cwarps * 32, csmem, ctx->stream>>>(ng, dnp, tp, tmpj, node_of, cap, nullptr, np32,
                                                                                            nj, d_status);
        ctx->launches++;
        gp = np32;
        gjs = nj;
        ns = nnj;
    }
    // symmetrise, unless the graph is its own transpose (every symmetric matrix at theta = 0)
    const uint32_t* gp32 = gp;
    const int32_t* gj = gjs;
    int* dasym = w.get<int>(1);
    DEV_ALLOC(dasym);
    DEV_TRY(cudaMemsetAsync(dasym, 0, sizeof(int), ctx->stream));
    symmetric_kernel<<<grid_rows(ng, 32), 256, 0, ctx->stream>>>(ng, gp, gjs, dasym);
    ctx->launches++;
    int asym = 0;
    rc = read_status(ctx, dasym, &asym);
    if (rc) return rc;
    if (asym) {
        // the transpose by column counts and cursors, its rows sorted, merged row by row
        uint32_t* tcnt = w.get<uint32_t>(ng + 1);
        uint32_t* tc = w.get<uint32_t>(ng + 1);
        uint32_t* cur = w.get<uint32_t>(ng + 1);
        int32_t* tj = w.get<int32_t>((int64_t)ns);
        uint32_t* sp32 = w.get<uint32_t>(ng + 1);
        DEV_ALLOC(tcnt && tc && cur && tj && sp32);
        DEV_TRY(cudaMemsetAsync(tcnt, 0, (ng + 1) * sizeof(uint32_t), ctx->stream));
        col_count_kernel<<<grid_rows((int64_t)ns, 256), 256, 0, ctx->stream>>>((int64_t)ns, gjs, tcnt);
        ctx->launches++;
        rc = scan_u32(ctx, tcnt, tc, ng, nullptr);
        if (rc) return rc;
        DEV_TRY(cudaMemcpyAsync(cur, tc, (ng + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
        transpose_fill_kernel<<<grid_rows(ng, 256), 256, 0, ctx->stream>>>(ng, gp, nullptr, gjs, nullptr, cur, tj, nullptr);
        ctx->launches++;
        rc = seg_sort(ctx, ng, tc, nullptr, tj, nullptr, d_status);
        if (rc) return rc;
        merge_kernel<<<grid_rows(ng, 256), 256, 0, ctx->stream>>>(ng, gp, gjs, tc, tj, cnt, nullptr, nullptr);
        ctx->launches++;
        uint64_t nsg = 0;
        rc = scan_u32(ctx, cnt, sp32, ng, &nsg);
        if (rc) return rc;
        int32_t* sj = w.get<int32_t>((int64_t)nsg);
        DEV_ALLOC(sj);
        merge_kernel<<<grid_rows(ng, 256), 256, 0, ctx->stream>>>(ng, gp, gjs, tc, tj, nullptr, sp32, sj);
        ctx->launches++;
        gp32 = sp32;
        gj = sj;
    }
    rc = read_status(ctx, d_status, &st);
    if (rc) return rc;
    if (st & kStOverflow) { *handoff = true; tm.handoff = nns ? 2 : 1; return FGPU_OK; }
    tm.graph += ms_since(tphase);
    tphase = clock::now();
    // aggregation: rounds of the distance-2 independent set, then the two assignment steps
    int8_t* mstate = w.get<int8_t>(ng);
    int8_t* mnext = w.get<int8_t>(ng);
    uint64_t* m1 = w.get<uint64_t>(ng);
    uint8_t* r1 = w.get<uint8_t>(ng);
    unsigned long long* dund = w.get<unsigned long long>(1);
    uint32_t* rflag = w.get<uint32_t>(ng + 1);
    uint32_t* rank = w.get<uint32_t>(ng + 1);
    int32_t* a1 = w.get<int32_t>(ng);
    int32_t* dagg_node = w.get<int32_t>(ng);
    DEV_ALLOC(mstate && mnext && m1 && r1 && dund && rflag && rank && a1 && dagg_node);
    const int gg = grid_rows(ng, 256);
    const int gm = grid_rows(ng, 256 / kMisLanes, 152 * 16);
    mis_init_kernel<<<gg, 256, 0, ctx->stream>>>(ng, gp32, mstate);
    ctx->launches++;
    for (int round = 0;; ++round) {
        if (round > 1000) { ctx->err = "gamg device set-up: aggregation did not converge"; return FGPU_ERR_INVALID; }
        DEV_TRY(cudaMemsetAsync(dund, 0, sizeof(unsigned long long), ctx->stream));
        mis_pass1_kernel<<<gm, 256, 0, ctx->stream>>>(ng, gp32, gj, mstate, m1, r1, round == 0);
        mis_pass2_kernel<<<gm, 256, 0, ctx->stream>>>(ng, gp32, gj, mstate, m1, r1, mnext, dund);
        ctx->launches += 2;
        std::swap(mstate, mnext);
        unsigned long long hund = 0;
        DEV_TRY(cudaMemcpyAsync(&hund, dund, sizeof(hund), cudaMemcpyDeviceToHost, ctx->stream));
        DEV_TRY(cudaStreamSynchronize(ctx->stream));
        if (hund == 0) break;
    }
    mis_root_flag_kernel<<<gg, 256, 0, ctx->stream>>>(ng, mstate, rflag);
    ctx->launches++;
    uint64_t nroots = 0;
    rc = scan_u32(ctx, rflag, rank, ng, &nroots);
    if (rc) return rc;
    mis_assign1_kernel<<<gg, 256, 0, ctx->stream>>>(ng, gp32, gj, mstate, rank, a1);
    mis_assign2_kernel<<<gg, 256, 0, ctx->stream>>>(ng, gp32, gj, mstate, a1, dagg_node);
    ctx->launches += 2;
    const int64_t nagg = (int64_t)nroots;
    std::vector<int32_t> agg_node;
    std::vector<int32_t>& hagg = nns ? agg_node : L.agg;
    hagg.resize(ng);
    DEV_TRY(cudaMemcpyAsync(hagg.data(), dagg_node, ng * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    DEV_TRY(cudaStreamSynchronize(ctx->stream));
    tm.aggregate += ms_since(tphase);
    tphase = clock::now();
    if (nagg == 0 || nagg >= ng) { *handoff = true; tm.handoff = 3; return FGPU_OK; }
    AmgDevCsr P0;
    double* ds0 = nullptr;
    int64_t ncoarse = nagg;
    if (nns) {
        // tentative prolongator from the near null space (host QR per aggregate, the host set-up's code)
        HostCsr hP0;
        if (amg_tentative_nns(*nns, agg_node, nagg, cfg.nthreads > 0 ? cfg.nthreads : 1, hP0, *next)) {
            ctx->err = "gamg: coarse level too large";
            return FGPU_ERR_INVALID;
        }
        if (hP0.ncols == 0 || hP0.ncols >= n) { *handoff = true; tm.handoff = 3; return FGPU_OK; }
        ncoarse = hP0.ncols;
        L.agg.assign(n, -1);
        for (int64_t I = 0; I < ng; ++I)
            for (int64_t i = nns->node_ptr[I]; i < nns->node_ptr[I + 1]; ++i) L.agg[i] = agg_node[I];
        rc = alloc_csr(ctx, P0, n, hP0.ncols, (int64_t)hP0.ja.size());
        if (rc) return rc;
        DEV_TRY(cudaMemcpyAsync(P0.ia, hP0.ia.data(), (n + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
        if (!hP0.ja.empty()) {
            DEV_TRY(cudaMemcpyAsync(P0.ja, hP0.ja.data(), hP0.ja.size() * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
            DEV_TRY(cudaMemcpyAsync(P0.a, hP0.a.data(), hP0.a.size() * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        }
        DEV_TRY(cudaStreamSynchronize(ctx->stream));            // hP0 is freed on leaving this block
    } else {
    // tentative prolongator (1/sqrt(|agg|), the host's 1.0 / std::sqrt of the exact size) and A P0
    const int32_t* dagg = dagg_node;
    unsigned int* dsz = w.get<unsigned int>(nagg);
    ds0 = w.get<double>(nagg);
    DEV_ALLOC(dsz && ds0);
    DEV_TRY(cudaMemsetAsync(dsz, 0, nagg * sizeof(unsigned int), ctx->stream));
    agg_size_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, dagg, dsz);
    agg_scale_kernel<<<grid_rows(nagg, 256), 256, 0, ctx->stream>>>(nagg, dsz, ds0);
    p0_count_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, dagg, cnt);
    ctx->launches += 3;
    uint64_t n0 = 0;
    rc = scan_u32(ctx, cnt, tp, n, &n0);
    if (rc) return rc;
    rc = alloc_csr(ctx, P0, n, nagg, (int64_t)n0);
    if (rc) return rc;
    p0_fill_kernel<<<grid_rows(n + 1, 256), 256, 0, ctx->stream>>>(n, dagg, ds0, tp, P0.ia, P0.ja, P0.a);
    ctx->launches++;
    }
    bool ovf = false;
    // lambda_max: wait for the Lanczos thread (A P0 does not need it)
    auto join_lanczos = [&]() -> int {
        const auto tw = clock::now();
        if (lanczos.joinable()) lanczos.join();
        ctx->launches += lz.launches;
        lz.launches = 0;
        tm.lanczos += ms_since(tw);
        if (lz.err != cudaSuccess) { ctx->err = std::string("gamg device set-up: lambda_max: ") + cudaGetErrorString(lz.err); return FGPU_ERR_CUDA; }
        L.lmax = lz.lmax;
        return FGPU_OK;
    };
    if (cfg.agg_smooths <= 0) {
        L.P = std::move(P0);
        rc = join_lanczos();
        if (rc) return rc;
    } else {
        AmgDevCsr AP0;
        rc = spgemm_dev(ctx, A, P0, AP0, d_status, &ovf, nns ? nullptr : dagg_node, ds0);
        if (rc) return rc;
        if (ovf) { *handoff = true; tm.handoff = 4; return FGPU_OK; }
        rc = join_lanczos();
        if (rc) return rc;
        const double omega = 4.0 / (3.0 * L.lmax);
        prolong_merge_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, P0.ia, P0.ja, P0.a, AP0.ia, AP0.ja, AP0.a, d, omega, cnt,
                                                                        nullptr, nullptr, nullptr);
        ctx->launches++;
        uint64_t pn = 0;
        rc = scan_u32(ctx, cnt, tp, n, &pn);
        if (rc) return rc;
        rc = alloc_csr(ctx, L.P, n, ncoarse, (int64_t)pn);
        if (rc) return rc;
        prolong_merge_kernel<<<grid_rows(n, 256), 256, 0, ctx->stream>>>(n, P0.ia, P0.ja, P0.a, AP0.ia, AP0.ja, AP0.a, d, omega, nullptr,
                                                                        tp, L.P.ja, L.P.a);
        u32_to_i64_kernel<<<grid_rows(n + 1, 256), 256, 0, ctx->stream>>>(n + 1, tp, L.P.ia);
        ctx->launches += 2;
        DEV_TRY(cudaStreamSynchronize(ctx->stream));         // P0 and A P0 are freed on leaving this block
    }
    rc = transpose_dev(ctx, L.P, L.R, d_status);
    if (rc) return rc;
    rc = read_status(ctx, d_status, &st);
    if (rc) return rc;
    if (st & kStOverflow) { *handoff = true; tm.handoff = 5; return FGPU_OK; }
    tm.prolong += ms_since(tphase);
    tphase = clock::now();
    // Galerkin product A_c = R (A P)
    AmgDevCsr AP;
    rc = spgemm_dev(ctx, A, L.P, AP, d_status, &ovf);
    if (rc) return rc;
    if (ovf) { *handoff = true; tm.handoff = 6; return FGPU_OK; }
    rc = spgemm_dev(ctx, L.R, AP, Ac, d_status, &ovf);
    if (rc) return rc;
    if (ovf) { *handoff = true; tm.handoff = 7; return FGPU_OK; }
    DEV_TRY(cudaStreamSynchronize(ctx->stream));             // the scratch of this level is freed on return
    tm.galerkin += ms_since(tphase);
    if ((double)ncoarse > 0.9 * (double)n) *last = true;
    return FGPU_OK;
}

}  // namespace

int amg_copy_to_host(fgpu_ctx* ctx, const AmgDevCsr& D, HostCsr& H) {
    H.nrows = D.nrows;
    H.ncols = D.ncols;
    H.ia.assign(D.nrows + 1, 0);
    H.ja.resize(D.nnz);
    H.a.resize(D.nnz);
    if (!D.ia) return FGPU_OK;
    DEV_TRY(cudaMemcpyAsync(H.ia.data(), D.ia, (D.nrows + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    if (D.nnz) {
        DEV_TRY(cudaMemcpyAsync(H.ja.data(), D.ja, D.nnz * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
        DEV_TRY(cudaMemcpyAsync(H.a.data(), D.a, D.nnz * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    }
    DEV_TRY(cudaStreamSynchronize(ctx->stream));
    return FGPU_OK;
}

int amg_build_device(fgpu_ctx* ctx, const fgpu_matrix* Am, const AmgHostCfg& cfg, AmgDevHierarchy& H, const AmgNns* nns) {
    const auto t0 = std::chrono::steady_clock::now();
    const int max_levels = cfg.max_levels > 0 ? cfg.max_levels : 10;
    const int64_t coarse_lim = cfg.coarse_eq_lim > 0 ? cfg.coarse_eq_lim : 800;
    H.levels.clear();
    H.tail = AmgHierarchy();
    int* d_status = nullptr;
    DEV_TRY(pool_malloc(ctx->stream, &d_status, sizeof(int)));
    struct StatusFree {
        int* p;
        ~StatusFree() { pool_free(p); }
    } status_free{d_status};
    DEV_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), ctx->stream));
    H.levels.emplace_back();
    {
        AmgDevCsr& A0 = H.levels[0].A;               // a view of the matrix's own arrays
        A0.own = false;
        A0.nrows = A0.ncols = Am->nrows;
        A0.nnz = Am->nnz;
        A0.ia = Am->d_ia;
        A0.ja = Am->d_ja;
        A0.a = static_cast<double*>(Am->d_val);
    }
    H.times = AmgSetupTimes();
    AmgNns cur;
    if (nns) cur = *nns;
    bool last = false;
    int l = 0;
    for (; l + 1 < max_levels && !last; ++l) {
        AmgDevLevel& L = H.levels[l];
        if (L.A.nrows <= coarse_lim || L.A.nrows <= kHandoffRows || L.A.nnz >= ((int64_t)1 << 32)) break;
        AmgDevCsr Ac;
        AmgNns next;
        bool handoff = false;
        const int rc = level_dev(ctx, L, cfg, nns ? &cur : nullptr, &next, d_status, Ac, &handoff, &last, H.times);
        if (rc) return rc;
        if (handoff) {
            DEV_TRY(cudaStreamSynchronize(ctx->stream));
            L.P = AmgDevCsr();
            L.R = AmgDevCsr();
            L.agg.clear();
            L.lmax = 0;
            DEV_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), ctx->stream));
            last = false;
            break;
        }
        H.levels.emplace_back();
        H.levels.back().A = std::move(Ac);
        if (nns) cur = std::move(next);
    }
    // the rest on the host, from level l (its operator copied)
    const auto t1 = std::chrono::steady_clock::now();
    HostCsr Al;
    int rc = amg_copy_to_host(ctx, H.levels[l].A, Al);
    if (rc) return rc;
    AmgHostCfg tc = cfg;
    tc.max_levels = last ? 1 : max_levels - l;
    std::string err;
    if (!amg_build_host(std::move(Al), tc, H.tail, err, nns ? &cur : nullptr)) { ctx->err = err; return FGPU_ERR_INVALID; }
    H.levels.resize(l);
    const auto t2 = std::chrono::steady_clock::now();
    H.times.total = std::chrono::duration<double, std::milli>(t2 - t0).count();
    H.times.tail = std::chrono::duration<double, std::milli>(t2 - t1).count();
    return FGPU_OK;
}

}  // namespace fgpu

namespace fgpu {

int amg_nns_from_cfg(fgpu_ctx* ctx, const fgpu_amg_cfg* cfg, int64_t n, AmgNns& nns, bool* has) {
    *has = false;
    if (!cfg || cfg->nns_count <= 0) return FGPU_OK;
    if (!cfg->nns || amg_nns_layout(cfg, n, nns)) { ctx->err = "gamg: invalid near null space (count, block size or vectors)"; return FGPU_ERR_INVALID; }
    std::vector<double> col(n);
    for (int j = 0; j < nns.m; ++j) {
        const fgpu_vector* v = cfg->nns[j];
        if (!v || v->n != n) { ctx->err = "gamg: a near null space vector does not match the matrix"; return FGPU_ERR_INVALID; }
        DEV_TRY(cudaMemcpyAsync(col.data(), v->d, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        DEV_TRY(cudaStreamSynchronize(ctx->stream));
        for (int64_t i = 0; i < n; ++i) nns.B[(size_t)i * nns.m + j] = col[i];
    }
    *has = true;
    return FGPU_OK;
}

}  // namespace fgpu

extern "C" int fgpu_space_rigid_body_modes(const fgpu_space* V, fgpu_vector* const* out) {
    using namespace fgpu;
    if (!V || !out) return FGPU_ERR_INVALID;
    fgpu_ctx* ctx = V->ctx;
    if (V->ncomp != 3 || V->mesh->cv != 4) { ctx->err = "rigid body modes: Pchv spaces on tetrahedral meshes only"; return FGPU_ERR_INVALID; }
    const int64_t nn = V->ndof / 3;
    for (int k = 0; k < 6; ++k)
        if (!out[k] || out[k]->n != V->ndof) { ctx->err = "rigid body modes: six vectors of the space's size"; return FGPU_ERR_INVALID; }
    std::vector<double> ref;
    if (!lagrange_nodes(V->order, ref) || (int)ref.size() != 3 * V->n) { ctx->err = "rigid body modes: orders 1-3"; return FGPU_ERR_INVALID; }
    std::vector<double> lam((size_t)V->n * 4);
    for (int a = 0; a < V->n; ++a) {                // barycentrics of the reference nodes ([-1, 1] reference tetrahedron)
        const double l1 = 0.5 * (1.0 + ref[a * 3]), l2 = 0.5 * (1.0 + ref[a * 3 + 1]), l3 = 0.5 * (1.0 + ref[a * 3 + 2]);
        lam[a * 4] = 1.0 - l1 - l2 - l3;
        lam[a * 4 + 1] = l1;
        lam[a * 4 + 2] = l2;
        lam[a * 4 + 3] = l3;
    }
    fgpu_mesh* M = V->mesh;
    if (M->h_xyz_stale) {
        DEV_TRY(cudaMemcpyAsync(M->h_xyz.data(), M->d_xyz, M->h_xyz.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        DEV_TRY(cudaStreamSynchronize(ctx->stream));
        M->h_xyz_stale = false;
    }
    double c[3] = {0.0, 0.0, 0.0};
    for (int64_t v = 0; v < M->nv; ++v)
        for (int d = 0; d < 3; ++d) c[d] += M->h_xyz[v * 3 + d];
    for (int d = 0; d < 3; ++d) c[d] /= (double)std::max<int64_t>(M->nv, 1);
    double *dlam = nullptr, *xn = nullptr;
    DEV_TRY(pool_malloc(ctx->stream, &dlam, lam.size() * sizeof(double)));
    struct Free { double*& a; double*& b; ~Free() { pool_free(a); pool_free(b); } } fr{dlam, xn};
    DEV_TRY(pool_malloc(ctx->stream, &xn, std::max<int64_t>(nn, 1) * 3 * sizeof(double)));
    DEV_TRY(cudaMemcpyAsync(dlam, lam.data(), lam.size() * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    node_coords_kernel<<<grid_rows(nn, 256), 256, 0, ctx->stream>>>(nn, V->n, V->d_inc_ptr, V->d_inc, M->d_tets, M->d_xyz, dlam, xn);
    rbm_kernel<<<grid_rows(nn, 256), 256, 0, ctx->stream>>>(nn, xn, c[0], c[1], c[2], out[0]->d, out[1]->d, out[2]->d, out[3]->d,
                                                           out[4]->d, out[5]->d);
    ctx->launches += 2;
    DEV_TRY(cudaGetLastError());
    DEV_TRY(cudaStreamSynchronize(ctx->stream));
    return FGPU_OK;
}

// ---------------------------------------------------------------------------------------------------
// The device-built hierarchy copied into the host set-up's inspection object (fgpu_amg_host_*), so
// that it can be compared with fgpu_amg_host_build's level by level.
// ---------------------------------------------------------------------------------------------------
extern "C" int fgpu_amg_device_build(fgpu_ctx* ctx, const fgpu_matrix* A, const fgpu_amg_cfg* cfg, fgpu_amg_host** out) {
    using namespace fgpu;
    if (!ctx || !A || !out) return FGPU_ERR_INVALID;
    *out = nullptr;
    if (A->precision != FGPU_F64) { ctx->err = "gamg: FP64 matrices only"; return FGPU_ERR_INVALID; }
    if (ctx->capturing) { ctx->err = "gamg: set-up is not capturable"; return FGPU_ERR_INVALID; }
    const AmgHostCfg hc = amg_host_cfg(cfg, ctx->host_threads);
    AmgNns nns;
    bool has_nns = false;
    int rc = amg_nns_from_cfg(ctx, cfg, A->nrows, nns, &has_nns);
    if (rc) return rc;
    AmgDevHierarchy D;
    rc = amg_build_device(ctx, A, hc, D, has_nns ? &nns : nullptr);
    if (rc) return rc;
    fgpu_amg_host* h = new fgpu_amg_host();
    for (auto& dl : D.levels) {
        h->H.levels.emplace_back();
        AmgHostLevel& hl = h->H.levels.back();
        if ((rc = amg_copy_to_host(ctx, dl.A, hl.A)) || (rc = amg_copy_to_host(ctx, dl.P, hl.P)) ||
            (rc = amg_copy_to_host(ctx, dl.R, hl.R))) {
            delete h;
            return rc;
        }
        hl.agg = dl.agg;
        hl.lmax = dl.lmax;
    }
    for (auto& tl : D.tail.levels) h->H.levels.push_back(std::move(tl));
    h->H.coarse_inv.swap(D.tail.coarse_inv);
    h->device_levels = (int)D.levels.size();
    *out = h;
    return FGPU_OK;
}

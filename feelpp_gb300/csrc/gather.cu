// Phase 2 of the two-phase assembly: every CSR entry is the sum, in element order, of its
// contributions in the element buffer (bilinearformcontext.hpp:784-847 -> MatSetValues
// ADD_VALUES adds element blocks in that order).
//
// The element matrices are symmetric and the buffer holds their upper triangles, so an entry (i, j)
// and its transpose are one sum: it is formed once and stored at both positions. The map of the sums
// is kept in slices (GatherPlan, built once per space):
//  * a sum (a pair of dofs i <= j) belongs to the bin of the first element that contributes to it
//    (a bin is a run of elements with about a thousand sums);
//  * inside a bin the sums are sorted by their number of contributions (descending), then by the
//    buffer index of the first one, and taken 32 at a time as slices: the lanes of a warp run the
//    same number of steps;
//  * the buffer keeps an element's entries grouped by the vertex, edge, face or cell that their two
//    dofs span (entry_order): the sums of one group have the same contributing elements, so
//    neighbouring lanes read neighbouring buffer entries at every step;
//  * a slice stores its indices step by step, 32 lanes side by side (soff: its first row of 32,
//    padding 0xFFFFFFFF): a step is one coalesced load of indices and one gather of values.
//
// What bounds it: sectors between L2 and the SMs, and DRAM. At P2 48^3 (25.8 M entries, 66 M
// contributions; ncu) 26 M load and 19 M store sectors, 568 MB read and 183 MB written, 0.159 ms with
// DRAM, L2 and L1 each at about 60 %. Before, one thread per entry walked the entry's own index list:
// 269 M warp instructions (the lanes of a warp have 1 to 24 contributions) against 112 M, 896 MB read,
// 0.275 ms. Sizes measured, gather phase before -> after: P2 64^3 0.640 -> 0.380 ms, P3 41x37x40
// 0.661 -> 0.465 ms, binary32 P2 47x50x49 0.192 -> 0.122 ms. Tried on the way: slices over all entries
// (no symmetry) with the sums staged in shared memory and stored in CSR order, 0.244 ms at P2 48^3
// (62 M load sectors: 8-byte values in scattered 32-byte sectors).
#include <algorithm>
#include <climits>
#include <string>
#include <type_traits>
#include <vector>

#include "df64.h"
#include "entries.h"
#include "fgpu_core.h"
#include "scan.cuh"
#include "asm_device.cuh"
#include "closed.cuh"

namespace fgpu {

namespace {

constexpr uint32_t kNoIndex = 0xFFFFFFFFu;

// Sum of the lane's contributions in steps r0 .. r1 - 1 of its slice, B steps' loads together; PIPE: the
// next batch's indices travel with this batch's values. df64: compensated sum in element order, the high
// parts through TwoSum, their rounding errors and the low parts in one binary32 accumulator, normalised
// once by the caller (error ~ (count) u^2 |sum|). binary32: a plain sum from -0 with -0 for absent terms, which
// changes no value and no sign; without a test per term the whole batch is loads and additions (P2 48^3 gather 117
// -> 114 us, P3 28^3 114 -> 105).
template <int MODE, int B, bool PIPE>
__device__ __forceinline__ float2 slice_sum(uint32_t r0, uint32_t r1, int lane, const uint32_t* __restrict__ sidx,
                                            const void* __restrict__ kbuf) {
    typedef typename std::conditional<MODE == kModeDF64, float2, float>::type V;
    const V* kb = reinterpret_cast<const V*>(kbuf);
    float sh = MODE == kModeDF64 ? 0.0f : -0.0f, sl = 0.0f;
    V none{};
    if constexpr (MODE == kModeF32) none = -0.0f;
    uint32_t ix[B];
    if (PIPE) {
#pragma unroll
        for (int u = 0; u < B; ++u) ix[u] = r0 + u < r1 ? __ldg(sidx + (size_t)(r0 + u) * 32 + lane) : kNoIndex;
    }
    for (uint32_t r = r0; r < r1; r += B) {
        V v[B];
        if (!PIPE) {
#pragma unroll
            for (int u = 0; u < B; ++u) ix[u] = r + u < r1 ? __ldg(sidx + (size_t)(r + u) * 32 + lane) : kNoIndex;
        }
#pragma unroll
        for (int u = 0; u < B; ++u) v[u] = ix[u] != kNoIndex ? __ldg(kb + ix[u]) : none;
        if (PIPE && r + B < r1) {
#pragma unroll
            for (int u = 0; u < B; ++u) ix[u] = r + B + u < r1 ? __ldg(sidx + (size_t)(r + B + u) * 32 + lane) : kNoIndex;
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if constexpr (MODE == kModeF32) {
                sh = f_add(sh, v[u]);
            } else if (r + u < r1) {
                const df t = two_sum(sh, v[u].x);
                sh = t.hi;
                sl = f_add(sl, f_add(t.lo, v[u].y));
            }
        }
    }
    return make_float2(sh, sl);
}

template <int MODE, bool ACC, class T>
__device__ __forceinline__ void store_sum(float2 v, T* __restrict__ val, uint32_t k0, uint32_t k1, T o0, T o1) {
    if constexpr (MODE == kModeDF64) {
        const df s = two_sum(v.x, v.y);
        if (ACC) {
            val[k0] = df2d(df_add(d2df(o0), s));
            if (k1 != kNoIndex) val[k1] = df2d(df_add(d2df(o1), s));
        } else {
            const double r = df2d(s);
            val[k0] = r;
            if (k1 != kNoIndex) val[k1] = r;
        }
    } else {
        val[k0] = ACC ? f_add(o0, v.x) : v.x;
        if (k1 != kNoIndex) val[k1] = ACC ? f_add(o1, v.x) : v.x;
    }
}

// one slice per warp; ACC: added to the values, which are loaded before the sum (a load after it would be one more
// round trip to memory at the end of the chain)
template <int MODE, int B, bool PIPE, bool ACC>
__device__ __forceinline__ void gather_slice(const GatherPlan& G, int64_t s, const void* __restrict__ kbuf, void* __restrict__ valv) {
    typedef typename std::conditional<MODE == kModeDF64, double, float>::type T;
    T* const val = reinterpret_cast<T*>(valv);
    const int lane = threadIdx.x & 31;
    const uint32_t r0 = __ldg(G.soff + s), r1 = __ldg(G.soff + s + 1);
    const uint32_t k0 = __ldg(G.pos0 + s * 32 + lane), k1 = __ldg(G.pos1 + s * 32 + lane);
    T o0 = 0, o1 = 0;
    if constexpr (ACC) {
        if (k0 != kNoIndex) {
            o0 = val[k0];
            if (k1 != kNoIndex) o1 = val[k1];
        }
    }
    const float2 v = slice_sum<MODE, B, PIPE>(r0, r1, lane, G.sidx, kbuf);
    if (k0 != kNoIndex) store_sum<MODE, ACC>(v, val, k0, k1, o0, o1);
}

template <int MODE, int B, bool PIPE, bool ACC>
__global__ void __launch_bounds__(256) gather_slices_kernel(GatherPlan G, const void* __restrict__ kbuf, void* __restrict__ valv) {
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < G.nslices; s += nw)
        gather_slice<MODE, B, PIPE, ACC>(G, s, kbuf, valv);
}

// the slices of all problems of a batch (slice_off: prefix sums of their slice counts)
template <int MODE, bool PIPE, bool ACC>
__global__ void __launch_bounds__(256) batch_gather_slices_kernel(int nprob, const BatchProblem* __restrict__ probs,
                                                                  const int64_t* __restrict__ slice_off, int64_t total) {
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= total) return;
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(slice_off + mid) <= s) lo = mid;
        else hi = mid - 1;
    }
    const BatchProblem& P = probs[lo];
    gather_slice<MODE, PIPE ? 8 : 4, PIPE, ACC>(P.plan, s - slice_off[lo], P.kbuf, P.val);
}

// a pair's block at its position k0 of the scalar pattern and its transpose at k1 (x: the values, acc: the same
// as double-float). ACC: added to the nine values of a block, loaded together (a load, a sum and a store in turn
// are nine round trips to memory one after another).
template <int MODE, bool ACC, class T>
__device__ __forceinline__ void elasticity_store(T* __restrict__ val, const int64_t* __restrict__ sia, const int32_t* __restrict__ ja,
                                                 uint32_t k0, uint32_t k1, const T (&x)[9], const df (&acc)[9]) {
    auto put = [&](uint32_t k, int32_t row, bool tr) {
        const int64_t s0 = sia[row];
        const int64_t len = sia[row + 1] - s0;
        T* const out = val + 9 * s0 + 3 * ((int64_t)k - s0);
        T old[9];
        if (ACC) {
#pragma unroll
            for (int q = 0; q < 9; ++q) old[q] = out[(q / 3) * 3 * len + q % 3];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                T* const o = out + c * 3 * len + d;
                const int q = tr ? d * 3 + c : c * 3 + d;
                if constexpr (!ACC) *o = x[q];
                else if constexpr (MODE == kModeDF64) *o = df2d(df_add(d2df(old[c * 3 + d]), acc[q]));
                else *o = f_add(old[c * 3 + d], x[q]);
            }
    };
    const int32_t j = __ldg(ja + k0), i = k1 == kNoIndex ? j : __ldg(ja + k1);
    put(k0, i, false);
    if (k1 != kNoIndex) put(k1, j, true);
}

// Vector elasticity: one lane per pair of nodes i <= j, its 3x3 block (row 3i+c, columns 3j+d) summed
// over the contributions in element order (bit 31 of an index: stored as (j, i), read transposed) and
// stored with its transpose at (j, i). sia, ja: the scalar pattern.
template <int MODE, int B, bool ACC>
__global__ void __launch_bounds__(128) gather_elasticity_slices_kernel(GatherPlan G, const int64_t* __restrict__ sia,
                                                                       const int32_t* __restrict__ ja, const void* __restrict__ kbuf,
                                                                       void* __restrict__ valv) {
    typedef typename std::conditional<MODE == kModeDF64, float2, float>::type V;
    const int lane = threadIdx.x & 31;
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= G.nslices) return;
    const uint32_t r0 = __ldg(G.soff + s), r1 = __ldg(G.soff + s + 1);
    const uint32_t k0 = __ldg(G.pos0 + s * 32 + lane), k1 = __ldg(G.pos1 + s * 32 + lane);
    // B contributions' blocks in flight, the next indices with them
    df acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = df{0.0f, 0.0f};
    uint32_t ix[B];
#pragma unroll
    for (int u = 0; u < B; ++u) ix[u] = r0 + u < r1 ? __ldg(G.sidx + (size_t)(r0 + u) * 32 + lane) : kNoIndex;
    for (uint32_t r = r0; r < r1; r += B) {
        V v[B][9];
        uint32_t cur[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            cur[u] = ix[u];
            const V* b = reinterpret_cast<const V*>(kbuf) + (size_t)(cur[u] & 0x7FFFFFFFu) * 9;
#pragma unroll
            for (int k = 0; k < 9; ++k) v[u][k] = cur[u] != kNoIndex ? __ldg(b + k) : V{};
        }
#pragma unroll
        for (int u = 0; u < B; ++u) ix[u] = r + B + u < r1 ? __ldg(G.sidx + (size_t)(r + B + u) * 32 + lane) : kNoIndex;
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if (cur[u] == kNoIndex) continue;
            const bool tr = (cur[u] & 0x80000000u) != 0;
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const V w = tr ? v[u][d * 3 + c] : v[u][c * 3 + d];
                    df& a = acc[c * 3 + d];
                    if constexpr (MODE == kModeDF64) a = r + u == r0 ? df{w.x, w.y} : df_add(a, df{w.x, w.y});
                    else a.hi = r + u == r0 ? w : f_add(a.hi, w);
                }
        }
    }
    if (k0 == kNoIndex) return;
    typedef typename std::conditional<MODE == kModeDF64, double, float>::type T;
    T* const val = reinterpret_cast<T*>(valv);
    T x[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        if constexpr (MODE == kModeDF64) x[k] = df2d(acc[k]);
        else x[k] = acc[k].hi;
    }
    elasticity_store<MODE, ACC>(val, sia, ja, k0, k1, x, acc);
}

// ---- vector elasticity without an element buffer ----
// With exact quadrature the tensor of a pair of functions is Y = sum n_kl u_k u_l^T over their barycentric
// derivatives (one for a vertex function, two for an edge function; p2_stiff_coef), u_a = (|T| / 5)^(1/2)
// grad l_a (P1: |T|^(1/2), n = 1), and lambda and mu enter after the sum over the elements:
// block = lambda Y + mu Y^T + mu tr(Y) 1.

// u_0 .. u_3 of each element: double-float, (hi, lo) of three coordinates and two words of padding each, so
// that a vector is one 32-byte sector (binary32: 16 bytes)
template <int MODE, int N>
__global__ void elasticity_vectors_kernel(int64_t nt, const double* __restrict__ xyz, const int32_t* __restrict__ tets,
                                          float4* __restrict__ rec, int* __restrict__ status) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nt; e += (int64_t)gridDim.x * blockDim.x) {
        const int4 t = *reinterpret_cast<const int4*>(tets + 4 * e);
        const double* X0 = xyz + 3 * (int64_t)t.x;
        const double* Xv[3] = {xyz + 3 * (int64_t)t.y, xyz + 3 * (int64_t)t.z, xyz + 3 * (int64_t)t.w};
        // cofactors and determinant in binary64 (30 operations): the vectors' error enters every entry
        double K[9];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) K[r * 3 + c] = Xv[c][r] - X0[r];
        const double C[9] = {K[4] * K[8] - K[5] * K[7], K[5] * K[6] - K[3] * K[8], K[3] * K[7] - K[4] * K[6],
                             K[2] * K[7] - K[1] * K[8], K[0] * K[8] - K[2] * K[6], K[1] * K[6] - K[0] * K[7],
                             K[1] * K[5] - K[2] * K[4], K[2] * K[3] - K[0] * K[5], K[0] * K[4] - K[1] * K[3]};
        const df J = d2df(0.125 * fabs(fma(K[0], C[0], fma(K[1], C[1], K[2] * C[2]))));
        if (!(J.hi > 0.0f) || !isfinite(J.hi)) atomicOr(status, kStatusBadElement);
        // grad l_a = C_a / (8 J), |T| = 4 J / 3: u = C_a / 4 (15 J)^(-1/2), P1 C_a / 4 (3 J)^(-1/2)
        const float m = N == 10 ? 15.0f : 3.0f;
        const df s = df_scale(df_rsqrt(df_mul(J, df{m, 0.0f})), 0.25f);
        df u[4][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
            for (int a = 1; a < 4; ++a) u[a][r] = df_mul(d2df(C[3 * r + a - 1]), s);
            const df v = two_sum(u[1][r].hi, u[2][r].hi), w = two_sum(v.hi, u[3][r].hi);
            u[0][r] = df_neg(two_sum(w.hi, f_add(f_add(v.lo, w.lo), f_add(f_add(u[1][r].lo, u[2][r].lo), u[3][r].lo))));
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (MODE == kModeDF64) {
                rec[8 * e + 2 * a] = make_float4(u[a][0].hi, u[a][0].lo, u[a][1].hi, u[a][1].lo);
                rec[8 * e + 2 * a + 1] = make_float4(u[a][2].hi, u[a][2].lo, 0.0f, 0.0f);
            } else {
                rec[4 * e + a] = make_float4(u[a][0].hi, u[a][1].hi, u[a][2].hi, 0.0f);
            }
        }
    }
}

// per entry of entry_order: the factors n_00, n_01, n_10, n_11 and its vectors (two bits each: a_0, a_1, b_0, b_1)
template <int N>
struct PairTable {
    float4 terms[N * (N + 1) / 2];
    uint32_t which[N * (N + 1) / 2];
};
template <int N>
constexpr PairTable<N> make_pair_table() {
    PairTable<N> P{};
    const EntryOrder O = make_entry_order(4, N == 10 ? 2 : 1, N);
    for (int t = 0; t < N * (N + 1) / 2; ++t) {
        const int i = O.a[t], j = O.b[t], ni = N == 10 ? bary_comps(i) : 1, nj = N == 10 ? bary_comps(j) : 1;
        for (int k = 0; k < 2; ++k) {
            P.which[t] |= (uint32_t)(N == 10 ? bary_comp(i, k < ni ? k : 0) : i) << (2 * k);
            P.which[t] |= (uint32_t)(N == 10 ? bary_comp(j, k < nj ? k : 0) : j) << (4 + 2 * k);
        }
        auto n = [&](int k, int l) { return k >= ni || l >= nj ? 0.0f : N == 10 ? (float)p2_stiff_coef(i, k, j, l) : 1.0f; };
        P.terms[t].x = n(0, 0);
        P.terms[t].y = n(0, 1);
        P.terms[t].z = n(1, 0);
        P.terms[t].w = n(1, 1);
    }
    return P;
}
__device__ const PairTable<4> kPairs1 = make_pair_table<4>();
__device__ const PairTable<10> kPairs2 = make_pair_table<10>();
template <int N>
__device__ __forceinline__ const PairTable<N>& pair_table() {
    if constexpr (N == 10) return kPairs2;
    else return kPairs1;
}

// One lane per pair of nodes i <= j (the slices of the scalar plan): Y summed over the pair's elements in
// element order, each from the element's vectors, then lambda and mu; stored with its transpose at (j, i).
// The 3x3 blocks of the element matrices (3 960 bytes per P2 element, 718 MB at 36x28x30) are never stored:
// 128 bytes of vectors are, which stay in L2, and a slice's lanes mostly share their elements, so that a
// step's loads are few sectors.
// Bound: FP32 issue half the time (18 compensated products and six two-term sums per contribution and lane,
// then the moduli and 18 stores per pair), the rest latency: pairs have three contributions on average. 64
// registers and two warps a block: 337 us, without the bound (72 registers) 372, two contributions in flight
// (96 registers) 405; fewer, longer-lived blocks 390-550 (neighbouring slices no longer run together). P2
// 36x28x30 in double-float: geometry 25, element blocks 413, gather 378 us -> vectors 15 and here 337; a pass
// 821 -> 372 us, P1 45^3 1070 -> 164 us, binary32 P2 20^3 193 -> 89 us. Error against
// binary64 5.7e-15 -> 5.1e-15.
template <int MODE, int N, int B, bool ACC>
__global__ void __launch_bounds__(64, 16) gather_elasticity_fused_kernel(GatherPlan G, const int64_t* __restrict__ sia,
                                                                      const int32_t* __restrict__ ja, const float4* __restrict__ rec,
                                                                      double lam, double mu, void* __restrict__ valv) {
    constexpr int NTRI = N * (N + 1) / 2;
    const PairTable<N>& pairs = pair_table<N>();
    const int lane = threadIdx.x & 31;
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= G.nslices) return;
    const uint32_t r0 = __ldg(G.soff + s), r1 = __ldg(G.soff + s + 1);
    const uint32_t k0 = __ldg(G.pos0 + s * 32 + lane), k1 = __ldg(G.pos1 + s * 32 + lane);
    float ys[9], ye[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) ys[k] = ye[k] = 0.0f;
    constexpr int NV = N == 10 ? 2 : 1, W = MODE == kModeDF64 ? 2 : 1;       // vectors per function; float4 per vector
    uint32_t ix[B];
#pragma unroll
    for (int u = 0; u < B; ++u) ix[u] = r0 + u < r1 ? __ldg(G.sidx + (size_t)(r0 + u) * 32 + lane) : kNoIndex;
    for (uint32_t r = r0; r < r1; r += B) {
        float4 va[B][NV * W], vb[B][NV * W];
        float4 pt[B];
        uint32_t cur[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            cur[u] = ix[u];
            const uint32_t idx = cur[u] == kNoIndex ? 0u : cur[u] & 0x7FFFFFFFu, e = idx / NTRI, t = idx - e * NTRI;
            uint32_t w = __ldg(&pairs.which[t]);
            pt[u] = __ldg(&pairs.terms[t]);
            if (cur[u] & 0x80000000u) {                              // stored as (j, i)
                w = (w >> 4 | w << 4) & 255u;
                const float x = pt[u].y;
                pt[u].y = pt[u].z;
                pt[u].z = x;
            }
            const float4* base = rec + (size_t)e * (4 * W);
#pragma unroll
            for (int q = 0; q < NV; ++q)
#pragma unroll
                for (int x = 0; x < W; ++x) {
                    va[u][q * W + x] = __ldg(base + (w >> (2 * q) & 3u) * W + x);
                    vb[u][q * W + x] = __ldg(base + (w >> (4 + 2 * q) & 3u) * W + x);
                }
        }
#pragma unroll
        for (int u = 0; u < B; ++u) ix[u] = r + B + u < r1 ? __ldg(G.sidx + (size_t)(r + B + u) * 32 + lane) : kNoIndex;
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if (cur[u] == kNoIndex) continue;
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                if constexpr (MODE == kModeDF64) {
                    auto vec = [](const float4* v, int c) {
                        return c == 0 ? df{v[0].x, v[0].y} : c == 1 ? df{v[0].z, v[0].w} : df{v[1].x, v[1].y};
                    };
                    df h[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if constexpr (N == 4) {
                            h[c] = vec(vb[u], c);
                        } else {
                            // n_q0 b_0 + n_q1 b_1, the factors small integers
                            const df b0 = vec(vb[u], c), b1 = vec(vb[u] + W, c);
                            const float n0 = q == 0 ? pt[u].x : pt[u].z, n1 = q == 0 ? pt[u].y : pt[u].w;
                            const float p0 = f_mul(n0, b0.hi), p1 = f_mul(n1, b1.hi);
                            float e = f_fma(n0, b0.lo, f_fma(n0, b0.hi, -p0));
                            e = f_fma(n1, b1.lo, f_add(e, f_fma(n1, b1.hi, -p1)));
                            const df x = two_sum(p0, p1);
                            h[c] = quick_two_sum(x.hi, f_add(x.lo, e));
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int d = 0; d < 3; ++d) df_dot_term(vec(va[u] + q * W, c), h[d], ys[3 * c + d], ye[3 * c + d]);
                } else {
                    auto vec = [](const float4& v, int c) { return c == 0 ? v.x : c == 1 ? v.y : v.z; };
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const float h = N == 4 ? vec(vb[u][0], d)
                                               : fmaf(q == 0 ? pt[u].x : pt[u].z, vec(vb[u][0], d), (q == 0 ? pt[u].y : pt[u].w) * vec(vb[u][NV - 1], d));
#pragma unroll
                        for (int c = 0; c < 3; ++c) ys[3 * c + d] = fmaf(vec(va[u][q], c), h, ys[3 * c + d]);
                    }
                }
            }
        }
    }
    if (k0 == kNoIndex) return;
    typedef typename std::conditional<MODE == kModeDF64, double, float>::type T;
    T* const val = reinterpret_cast<T*>(valv);
    df acc[9];
    T x[9];
    if constexpr (MODE == kModeDF64) {
        const df l = d2df(lam), m = d2df(mu);
        df y[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) y[k] = two_sum(ys[k], ye[k]);
        const df mtr = df_mul(m, df_add(df_add(y[0], y[4]), y[8]));
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                df v = df_add(df_mul(l, y[c * 3 + d]), df_mul(m, y[d * 3 + c]));
                if (c == d) v = df_add(v, mtr);
                acc[c * 3 + d] = v;
                x[c * 3 + d] = df2d(v);
            }
    } else {
        const float l = (float)lam, m = (float)mu, tr = ys[0] + ys[4] + ys[8];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float v = fmaf(l, ys[c * 3 + d], m * ys[d * 3 + c]);
                if (c == d) v = fmaf(m, tr, v);
                x[c * 3 + d] = v;
                acc[c * 3 + d] = df{v, 0.0f};
            }
    }
    elasticity_store<MODE, ACC>(val, sia, ja, k0, k1, x, acc);
}

// the values of the matrix to a mapped page-locked host buffer
__global__ void __launch_bounds__(256) values_to_host_kernel(int64_t nnz, const double* __restrict__ val, double* __restrict__ hout) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x) hout[k] = val[k];
}

// lowest[c]: the lowest row that part c of the slices writes to (the row of a position is the column of its
// transpose's)
__global__ void __launch_bounds__(256) part_rows_kernel(GatherPlan G, int parts, const int32_t* __restrict__ ja, int* __restrict__ lowest) {
    const int64_t q = (G.nslices + parts - 1) / parts, n = G.nslices * 32;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k0 = G.pos0[k], k1 = G.pos1[k];
        int r = k0 == kNoIndex ? INT_MAX : k1 == kNoIndex ? ja[k0] : min(ja[k0], ja[k1]);
        r = __reduce_min_sync(0xffffffffu, r);
        if ((threadIdx.x & 31) == 0 && r != INT_MAX) atomicMin(lowest + (k >> 5) / q, r);
    }
}

// ---- the plan (once per space) ----

// The space's tables that the plan is built from; tri: pair (a, b) of local dofs -> buffer entry.
struct PlanIn {
    int64_t nrows;
    uint32_t n, ntri;
    int bin_shift, mark;                  // a bin is 2^bin_shift elements
    const int64_t* ia;
    const int64_t* inc_ptr;
    const int32_t* inc;
    const int32_t* l2n;
    const uint8_t* pos;
    const uint16_t* tri;
};

// One warp per row r, its incident elements in element order, 32 / n of them at a time with one lane
// per element dof; the dofs j >= r are the row's sums. first[idx], idx a buffer entry: the sum whose
// first contribution it is (0: none).
// FILL 0: first[idx] = the sum's number of contributions (counted in any order; the first by minimum).
// FILL 1: first[idx] holds 1 + the sum's place in its bin; the sum's CSR positions and the buffer
// indices of its steps, in element order.
// mark: bit 31 of an index whose element entry is stored as (j, i).
template <int FILL, int U>
__global__ void __launch_bounds__(256, 6) plan_walk_kernel(PlanIn in, uint16_t* __restrict__ first, const uint32_t* __restrict__ slice0,
                                                        const uint32_t* __restrict__ soff, uint32_t* __restrict__ pos0,
                                                        uint32_t* __restrict__ pos1, uint32_t* __restrict__ sidx,
                                                        int* __restrict__ status) {
    __shared__ uint32_t at[8][256];     // 0: first buffer entry; 1: place of the sum's next step
    __shared__ uint32_t cnt[FILL ? 1 : 8][256];
    __shared__ uint16_t tri[32 * 32];   // n <= 32 (checked by the launcher)
    const uint32_t n = in.n;
    for (uint32_t k = threadIdx.x; k < n * n; k += blockDim.x) tri[k] = in.tri[k];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int epw = 32 / (int)n, grp = lane / (int)n, lj = lane - grp * (int)n;
    // (32-bit indices: fewer than 2^32 contributions, checked by the launcher)
    for (uint32_t r = blockIdx.x * 8 + warp; r < (uint32_t)in.nrows; r += gridDim.x * 8) {
        const int64_t start = in.ia[r];
        const int len = (int)(in.ia[r + 1] - start);
        if (len > 256) {
            if (lane == 0) atomicOr(status, kStatusRowOverflow);
            continue;
        }
        if (!FILL)
            for (int k = lane; k < len; k += 32) {
                at[warp][k] = kNoIndex;
                cnt[FILL ? 0 : warp][k] = 0;
            }
        __syncwarp();
        // U = 2 steps' loads together: the chain of a step is up to five dependent loads, its work a few
        // instructions (P2 64^3 fill 1.36 ms, 1.47 a step at a time; U = 4 at P3 1.54 against 1.29; rows
        // pipelined over iterations 2.7 ms: fewer warps per SM)
        const uint32_t t1 = (uint32_t)in.inc_ptr[r + 1];
        for (uint32_t t = (uint32_t)in.inc_ptr[r]; t < t1; t += U * epw) {
            uint32_t code[U], idx[U], w0[U];
            int32_t j[U];
            int p[U];
            bool on[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                on[u] = grp < epw && t + u * epw + grp < t1;
                code[u] = on[u] ? (uint32_t)in.inc[t + u * epw + grp] : 0u;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t e = code[u] >> 5, li = code[u] & 31u;
                j[u] = on[u] ? in.l2n[e * n + lj] : -1;
                p[u] = on[u] ? in.pos[(e * n + li) * n + lj] : 0;
                idx[u] = e * in.ntri + (on[u] ? tri[li * n + lj] : 0u);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                on[u] = on[u] && (uint32_t)j[u] >= r;
                w0[u] = FILL && on[u] ? first[idx[u]] : 0u;
            }
            if (FILL) {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (w0[u]) {                   // the sum's first contribution: its positions and its place
                        const uint32_t e = code[u] >> 5, li = code[u] & 31u;
                        const uint32_t slot = slice0[e >> in.bin_shift] * 32 + w0[u] - 1;
                        at[warp][p[u]] = soff[slot >> 5] * 32 + (slot & 31);
                        pos0[slot] = (uint32_t)start + p[u];
                        pos1[slot] = (uint32_t)j[u] != r ? (uint32_t)in.ia[j[u]] + in.pos[(e * n + lj) * n + li] : kNoIndex;
                    }
                __syncwarp();
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!FILL) {
                    if (on[u]) {
                        atomicAdd(&cnt[FILL ? 0 : warp][p[u]], 1u);
                        atomicMin(&at[warp][p[u]], idx[u]);
                    }
                } else {
                    // places in element order: the step's elements one after another (their dofs are distinct)
                    uint32_t w = 0;
                    for (int g = 0; g < epw; ++g) {
                        if (on[u] && g == grp) {
                            w = at[warp][p[u]];
                            at[warp][p[u]] = w + 32;
                        }
                        __syncwarp();
                    }
                    if (on[u]) sidx[w] = idx[u] | (in.mark && (code[u] & 31u) > (uint32_t)lj ? 0x80000000u : 0u);
                }
            }
            __syncwarp();
        }
        if (!FILL)
            for (int k = lane; k < len; k += 32) {
                const uint32_t c = cnt[FILL ? 0 : warp][k];
                if (c) first[at[warp][k]] = (uint16_t)min(c, 0xFFFFu);
            }
        __syncwarp();
    }
}

// sums of each bin (one warp per bin, eight counts per load; a bin starts at a multiple of `per`)
__global__ void __launch_bounds__(256) bin_count_kernel(int64_t nbins, int64_t total, int per, const uint16_t* __restrict__ first,
                                                        uint32_t* __restrict__ cnt) {
    const int64_t bin = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (bin >= nbins) return;
    const int lane = threadIdx.x & 31;
    const int64_t b = bin * per, e = b + per < total ? b + per : total;
    const int64_t b8 = (b + 7) & ~(int64_t)7, e8 = e & ~(int64_t)7;
    uint32_t c = 0;
    if (b8 < e8) {
        for (int64_t k = b8 + 8 * lane; k < e8; k += 256) {
            const uint4 v = *reinterpret_cast<const uint4*>(first + k);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) c += ((w[u] & 0xFFFFu) != 0) + ((w[u] >> 16) != 0);
        }
        if (b + lane < b8) c += first[b + lane] != 0;
        if (e8 + lane < e) c += first[e8 + lane] != 0;
    } else {
        for (int64_t k = b + lane; k < e; k += 32) c += first[k] != 0;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) cnt[bin] = c;
}

// one block: the first slice of every bin, and the number of slices
__global__ void __launch_bounds__(1024) bin_scan_kernel(int64_t nbins, const uint32_t* __restrict__ cnt, uint32_t* __restrict__ slice0,
                                                        unsigned long long* __restrict__ total) {
    __shared__ unsigned long long part[1024];
    unsigned long long run = 0;
    for (int64_t b0 = 0; b0 < nbins; b0 += 4096) {          // four consecutive bins per thread
        const int64_t k0 = b0 + 4 * threadIdx.x;
        uint32_t c[4];
        unsigned long long t = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            c[u] = k0 + u < nbins ? (cnt[k0 + u] + 31) / 32 : 0u;
            t += c[u];
        }
        part[threadIdx.x] = t;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            const unsigned long long v = threadIdx.x >= (unsigned)o ? part[threadIdx.x - o] : 0ull;
            __syncthreads();
            part[threadIdx.x] += v;
            __syncthreads();
        }
        unsigned long long x = run + part[threadIdx.x] - t;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + u < nbins) {
                slice0[k0 + u] = (uint32_t)x;
                x += c[u];
            }
        run += part[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = run;
}

// One block per bin: the places of its sums by a stable counting sort (contributions descending, then
// buffer entry), written over the counts as place + 1, and each slice's number of steps (zero before). Most
// entries are zero (P3: five of six): the counts are read eight at a time and those of 2048 entries compacted
// first (256 entries at a time before: P2 64^3 273 -> 210 us, P3 41x37x40 275 -> 249).
__global__ void __launch_bounds__(256) bin_rank_kernel(int64_t total, int per, uint16_t* __restrict__ first, const uint32_t* __restrict__ slice0,
                                                       uint32_t* __restrict__ steps) {
    __shared__ uint32_t off[256];       // by class min(contributions, 255): next place
    __shared__ uint16_t wcnt[8][256];   // the class's sums in each warp's part of a batch
    __shared__ uint32_t list[2048];     // entry (upper half) and contributions of the sums of a chunk
    __shared__ uint32_t part[256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t base = (int64_t)blockIdx.x * per;
    const int cnt = (int)(total - base < per ? total - base : per);
    auto load8 = [&](int k, uint32_t (&c)[8]) {          // counts of entries k .. k + 7, zero past the bin
        if (k + 8 <= cnt && (per & 7) == 0) {
            const uint4 v = *reinterpret_cast<const uint4*>(first + base + k);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = u & 1 ? w[u >> 1] >> 16 : w[u >> 1] & 0xFFFFu;
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = k + u < cnt ? first[base + k + u] : 0u;
        }
    };
    off[tid] = 0;
    for (int k = tid; k < 8 * 256; k += 256) (&wcnt[0][0])[k] = 0;
    __syncthreads();
    for (int k = 8 * tid; k < cnt; k += 8 * 256) {
        uint32_t c[8];
        load8(k, c);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c[u]) atomicAdd(&off[min(c[u], 255u)], 1u);
    }
    __syncthreads();
    // exclusive sums from the largest class down
    const uint32_t own = off[255 - tid];
    part[tid] = own;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {
        const uint32_t v = tid >= o ? part[tid - o] : 0u;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    off[255 - tid] = part[tid] - own;
    __syncthreads();
    for (int b0 = 0; b0 < cnt; b0 += 2048) {
        // the chunk's sums in order
        uint32_t c8[8];
        load8(b0 + 8 * tid, c8);
        uint32_t nz = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) nz += c8[u] != 0;
        uint32_t x = nz;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[warp] = x;
        __syncthreads();
        uint32_t at = x - nz, sums = 0;
        for (int w = 0; w < 8; ++w) {
            if (w < warp) at += part[w];
            sums += part[w];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c8[u]) list[at++] = (uint32_t)(b0 + 8 * tid + u) << 16 | c8[u];
        __syncthreads();
        for (uint32_t l0 = 0; l0 < sums; l0 += 256) {
            const uint32_t item = l0 + tid < sums ? list[l0 + tid] : 0u, c = item & 0xFFFFu, cls = min(c, 255u);
            const unsigned same = __match_any_sync(0xffffffffu, cls);
            const bool leader = c && lane == __ffs(same) - 1;
            if (leader) wcnt[warp][cls] = (uint16_t)__popc(same);
            __syncthreads();
            if (c) {
                uint32_t place = off[cls] + __popc(same & ((1u << lane) - 1u));
                for (int w = 0; w < warp; ++w) place += wcnt[w][cls];
                first[base + (item >> 16)] = (uint16_t)(place + 1);
                if ((place & 31) == 0 || cls == 255u) atomicMax(steps + slice0[blockIdx.x] + (place >> 5), c);
            }
            __syncthreads();
            if (leader) {
                atomicAdd(&off[cls], (uint32_t)__popc(same));
                wcnt[warp][cls] = 0;
            }
            __syncthreads();
        }
    }
}

int sm_count(const fgpu_ctx* ctx) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    return std::max(sms, 1);
}

// All slices resident at once (64 warps per SM): the kernel lasts as long as its longest chain of loads,
// which the pipelined sum shortens (P1 10x9x11: 3.8 against 6.2 us); where warps queue, the plain sum's
// fewer instructions win (P2 64^3: 0.380 against 0.400 ms).
bool one_wave(const fgpu_ctx* ctx, int64_t nslices) { return nslices <= 64 * (int64_t)sm_count(ctx); }

template <int FILL>
void launch_walk(fgpu_ctx* ctx, int blocks, const PlanIn& in, uint16_t* first, const uint32_t* slice0, const uint32_t* soff,
                 uint32_t* pos0, uint32_t* pos1, uint32_t* sidx) {
    plan_walk_kernel<FILL, 2><<<blocks, 256, 0, ctx->stream>>>(in, first, slice0, soff, pos0, pos1, sidx, ctx->d_status);
}

template <int MODE, bool PIPE, bool ACC>
void launch_slices(fgpu_ctx* ctx, const fgpu_matrix* A, const GatherPlan& G, int threads, int bpsm, int batch) {
    const int64_t need = (G.nslices + threads / 32 - 1) / (threads / 32);
    const int blocks = (int)std::max<int64_t>(1, bpsm > 0 ? std::min<int64_t>(need, (int64_t)sm_count(ctx) * bpsm) : need);
    switch (batch) {
        case 2: gather_slices_kernel<MODE, 2, PIPE, ACC><<<blocks, threads, 0, ctx->stream>>>(G, A->d_kbuf, A->d_val); break;
        case 8: gather_slices_kernel<MODE, 8, PIPE, ACC><<<blocks, threads, 0, ctx->stream>>>(G, A->d_kbuf, A->d_val); break;
        default: gather_slices_kernel<MODE, 4, PIPE, ACC><<<blocks, threads, 0, ctx->stream>>>(G, A->d_kbuf, A->d_val); break;
    }
}

}  // namespace

// the order as pairs a * 256 + b (a <= b)
std::vector<uint16_t> entry_order(int cell_vertices, int order, int n) {
    const EntryOrder E = make_entry_order(cell_vertices, order, n);
    std::vector<uint16_t> out;
    for (int t = 0; t < E.ntri; ++t) out.push_back((uint16_t)(E.a[t] * 256 + E.b[t]));
    return out;
}

void gather_plan_free(fgpu_space* V) {
    cudaFree(V->plan.pos0);
    cudaFree(V->plan.sidx);
    V->plan = GatherPlan{};
}

bool gather_plan_ready(const fgpu_space* V) { return V->plan.sidx != nullptr; }

// Device memory of the map while it is built, in bytes (nt elements, n local dofs).
size_t gather_plan_bytes(int64_t nt, int n, int64_t nnz) { return (size_t)nt * n * (n + 1) / 2 * 7 + (size_t)nnz * 6 + (size_t)nt * 300; }

int launch_build_gather_map(fgpu_ctx* ctx, fgpu_space* V) {
    if (gather_plan_ready(V)) return FGPU_OK;
    const DevPattern& P = *V->pattern;
    const int n = V->n, ntri = n * (n + 1) / 2;
    const int64_t nt = V->mesh->nt, nnz = P.nnz, entries = nt * ntri;
    if (nt * (int64_t)n * n >= (int64_t)UINT32_MAX || entries >= ((int64_t)1 << 31)) {
        ctx->err = "gather map: more than 2^32 contributions or 2^31 buffered entries";
        return FGPU_ERR_INVALID;
    }
    if (!V->d_pos) { ctx->err = "gather map: no position table"; return FGPU_ERR_INVALID; }
    if (n > 32) { ctx->err = "gather map: more than 32 local dofs"; return FGPU_ERR_INVALID; }
    const std::vector<uint16_t> ab = entry_order(V->mesh->cv, V->order, n);
    std::vector<uint16_t> tri((size_t)n * n);
    for (int t = 0; t < ntri; ++t) tri[(ab[t] >> 8) * n + (ab[t] & 255)] = tri[(ab[t] & 255) * n + (ab[t] >> 8)] = (uint16_t)t;
    // elements per bin: about a thousand sums on average, fewer than 2^16 buffer entries
    int shift = 0;
    while ((2 << shift) * ntri < 65536 && nnz / 2 * (2 << shift) <= 1400 * nt) ++shift;
    const int per_bin = 1 << shift;
    const int64_t nbins = (nt + per_bin - 1) / per_bin;
    const int64_t max_slices = (nnz + P.nrows) / 64 + nbins + 1;     // a sum per pair i <= j, one partial slice per bin
    const int sms = sm_count(ctx);
    // scratch in one block (from the pool: cudaMalloc and cudaFree of it were 160 of the 410 us of a first P2
    // pass over 14x13x15 boxes): totals, scan sums, bins, steps, the first contributions, the pair table
    const size_t s_tot = 16, s_sum = (scan_chunks(max_slices) + 1) * 8, s_bin = (size_t)nbins * 8, s_step = (size_t)max_slices * 4,
                 s_first = ((size_t)entries * 2 + 15) & ~(size_t)15;
    char* scratch = nullptr;
    GatherPlan G{};
    cudaError_t e = pool_malloc(ctx->stream, &scratch, s_tot + s_sum + s_bin + s_step + 16 + s_first + tri.size() * 2);
    unsigned long long* d_total = reinterpret_cast<unsigned long long*>(scratch);
    unsigned long long* sums = d_total + 2;
    uint32_t *cnt = reinterpret_cast<uint32_t*>(scratch + s_tot + s_sum), *slice0 = cnt + nbins, *steps = slice0 + nbins;
    uint16_t* first = reinterpret_cast<uint16_t*>(scratch + ((s_tot + s_sum + s_bin + s_step + 15) & ~(size_t)15));
    uint16_t* d_tri = reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(first) + s_first);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_tri, tri.data(), tri.size() * sizeof(uint16_t), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(first, 0, (size_t)entries * sizeof(uint16_t), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(steps, 0, s_step, ctx->stream);
    const PlanIn in{P.nrows, (uint32_t)n, (uint32_t)ntri, shift, V->ncomp > 1, P.d_ia, V->d_inc_ptr, V->d_inc, V->d_l2n, V->d_pos, d_tri};
    const int walkers = (int)std::max<int64_t>(1, std::min<int64_t>((P.nrows + 7) / 8, (int64_t)sms * 64));
    if (e == cudaSuccess) {
        launch_walk<0>(ctx, walkers, in, first, nullptr, nullptr, nullptr, nullptr, nullptr);
        bin_count_kernel<<<(int)((nbins + 7) / 8), 256, 0, ctx->stream>>>(nbins, entries, per_bin * ntri, first, cnt);
        bin_scan_kernel<<<1, 1024, 0, ctx->stream>>>(nbins, cnt, slice0, d_total);
        bin_rank_kernel<<<(int)nbins, 256, 0, ctx->stream>>>(entries, per_bin * ntri, first, slice0, steps);
        ctx->launches += 4;
        e = cudaGetLastError();
    }
    const size_t slots = (size_t)max_slices * 32;
    if (e == cudaSuccess) e = dev_malloc(&G.pos0, (2 * slots + max_slices + 1) * sizeof(uint32_t));
    G.pos1 = G.pos0 + slots;
    G.soff = G.pos1 + slots;
    if (e == cudaSuccess) e = cudaMemsetAsync(G.pos0, 0xFF, slots * sizeof(uint32_t), ctx->stream);   // (pos1: written with pos0)
    if (e == cudaSuccess) {
        scan_u32_launch(ctx, steps, G.soff, max_slices, sums);
        e = cudaGetLastError();
    }
    unsigned long long nslices = 0, rows = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&nslices, d_total, sizeof(nslices), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&rows, sums + scan_chunks(max_slices), sizeof(rows), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    G.nslices = (int64_t)nslices;
    const size_t words = std::max<size_t>(1, (size_t)rows * 32);
    int rc = FGPU_OK;
    if (e == cudaSuccess && words > 0xFFFFFFFFull) {
        ctx->err = "gather map: more than 2^32 padded contributions";
        rc = FGPU_ERR_INVALID;
    }
    if (e == cudaSuccess && rc == FGPU_OK) e = dev_malloc(&G.sidx, words * sizeof(uint32_t));
    if (e == cudaSuccess && rc == FGPU_OK) e = cudaMemsetAsync(G.sidx, 0xFF, words * sizeof(uint32_t), ctx->stream);
    if (e == cudaSuccess && rc == FGPU_OK) {
        launch_walk<1>(ctx, walkers, in, first, slice0, G.soff, G.pos0, G.pos1, G.sidx);
        ctx->launches++;
        e = cudaGetLastError();
    }
    pool_free(scratch);              // (in stream order: the walk runs on while the caller allocates and launches)
    if (e != cudaSuccess || rc != FGPU_OK) {
        cudaFree(G.pos0); cudaFree(G.sidx);
        if (rc) return rc;
        cudaGetLastError();
        ctx->err = std::string("gather map: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? FGPU_ERR_ALLOC : FGPU_ERR_CUDA;
    }
    V->plan = G;
    return FGPU_OK;
}

void launch_gather_slices(fgpu_ctx* ctx, const fgpu_matrix* A, int threads, int bpsm, int batch, int pipe, int accumulate) {
    const GatherPlan& G = A->space->plan;
    if (accumulate) {                // (the shapes are timed on plain assemblies)
        pipe = one_wave(ctx, G.nslices);
        threads = 256;
        bpsm = 0;
        batch = pipe ? 8 : 4;
    }
#define SLICES(MODE, PIPE)                                                             \
    do {                                                                               \
        if (accumulate) launch_slices<MODE, PIPE, true>(ctx, A, G, threads, bpsm, batch);  \
        else launch_slices<MODE, PIPE, false>(ctx, A, G, threads, bpsm, batch);            \
    } while (0)
    if (A->precision == FGPU_F32) {
        if (pipe) SLICES(kModeF32, true); else SLICES(kModeF32, false);
    } else {
        if (pipe) SLICES(kModeDF64, true); else SLICES(kModeDF64, false);
    }
#undef SLICES
}

int launch_gather_phase(fgpu_ctx* ctx, fgpu_matrix* A, int accumulate) {
    PendingEvent ev;
    prof_begin(ctx, "assemble_gather", ev);
    if (one_wave(ctx, A->space->plan.nslices)) launch_gather_slices(ctx, A, 256, 0, 8, 1, accumulate);
    else launch_gather_slices(ctx, A, 256, 0, 4, 0, accumulate);
    prof_end(ctx, ev);
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    return FGPU_OK;
}

int launch_gather_elasticity(fgpu_ctx* ctx, const fgpu_matrix* A, int accumulate) {
    const GatherPlan& G = A->space->plan;
    const DevPattern& P = *A->pattern;
    const int blocks = (int)std::max<int64_t>(1, (G.nslices + 3) / 4);
    PendingEvent ev;
    prof_begin(ctx, "assemble_gather_elasticity", ev);
    // two blocks in flight per lane (P2 36x28x30: 0.378 ms, 0.635 one at a time); six where every slice is
    // resident and the longest chain, a vertex's 24 blocks, is what counts (P1 8^3: 48 against 56 us a pass)
#define EL_GATHER(MODE, B)                                                                                                 \
    do {                                                                                                                   \
        if (accumulate) gather_elasticity_slices_kernel<MODE, B, true><<<blocks, 128, 0, ctx->stream>>>(G, P.d_ia, P.d_ja, A->d_kbuf, A->d_val);  \
        else gather_elasticity_slices_kernel<MODE, B, false><<<blocks, 128, 0, ctx->stream>>>(G, P.d_ia, P.d_ja, A->d_kbuf, A->d_val);            \
    } while (0)
    if (one_wave(ctx, G.nslices)) {
        if (A->precision == FGPU_F32) EL_GATHER(kModeF32, 6); else EL_GATHER(kModeDF64, 6);
    } else {
        if (A->precision == FGPU_F32) EL_GATHER(kModeF32, 2); else EL_GATHER(kModeDF64, 2);
    }
#undef EL_GATHER
    prof_end(ctx, ev);
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    return FGPU_OK;
}

// rec: 128 bytes per element
int launch_gather_elasticity_fused(fgpu_ctx* ctx, const fgpu_matrix* A, double lam, double mu, float4* rec, int accumulate) {
    const GatherPlan& G = A->space->plan;
    const DevPattern& P = *A->pattern;
    const fgpu_mesh* M = A->space->mesh;
    const bool f32 = A->precision == FGPU_F32, p2 = A->space->order == 2;
    PendingEvent ev;
    prof_begin(ctx, "geometry", ev);
    const int gb = (int)std::max<int64_t>(1, std::min<int64_t>((M->nt + 127) / 128, 152 * 16));
#define EL_VECTORS(MODE, N) elasticity_vectors_kernel<MODE, N><<<gb, 128, 0, ctx->stream>>>(M->nt, M->d_xyz, M->d_tets, rec, ctx->d_status)
    if (p2) { if (f32) EL_VECTORS(kModeF32, 10); else EL_VECTORS(kModeDF64, 10); }
    else { if (f32) EL_VECTORS(kModeF32, 4); else EL_VECTORS(kModeDF64, 4); }
#undef EL_VECTORS
    prof_end(ctx, ev);
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    const int blocks = (int)std::max<int64_t>(1, (G.nslices + 1) / 2);
    prof_begin(ctx, "assemble_gather_elasticity", ev);
#define EL_GATHER(MODE, N, B)                                                                                              \
    do {                                                                                                                   \
        if (accumulate) gather_elasticity_fused_kernel<MODE, N, B, true><<<blocks, 64, 0, ctx->stream>>>(G, P.d_ia, P.d_ja, rec, lam, mu, A->d_val);  \
        else gather_elasticity_fused_kernel<MODE, N, B, false><<<blocks, 64, 0, ctx->stream>>>(G, P.d_ia, P.d_ja, rec, lam, mu, A->d_val);            \
    } while (0)
    if (p2) { if (f32) EL_GATHER(kModeF32, 10, 2); else EL_GATHER(kModeDF64, 10, 1); }
    else { if (f32) EL_GATHER(kModeF32, 4, 4); else EL_GATHER(kModeDF64, 4, 2); }
#undef EL_GATHER
    prof_end(ctx, ev);
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    return FGPU_OK;
}

// The host assembly's parts, once per space. The ends are rounded down to whole lines of 512 bytes: a part that starts
// anywhere makes partial writes of its stores to the host (P2 64^3 by kernel stores: 3.67 against 3.02 ms).
int plan_parts(fgpu_ctx* ctx, fgpu_space* V, int parts) {
    const GatherPlan& G = V->plan;
    HostParts& H = V->host_parts;
    if (H.count == parts) return FGPU_OK;
    const DevPattern& P = *V->pattern;
    int* lowest = nullptr;
    FGPU_CUDA_CHECK(ctx, pool_malloc(ctx->stream, &lowest, kHostParts * sizeof(int)));
    struct Free { int* p; ~Free() { pool_free(p); } } fr{lowest};
    int h[kHostParts];
    FGPU_CUDA_CHECK(ctx, cudaMemsetAsync(lowest, 0x7F, sizeof(h), ctx->stream));
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((G.nslices * 32 + 255) / 256, (int64_t)sm_count(ctx) * 16));
    part_rows_kernel<<<(int)blocks, 256, 0, ctx->stream>>>(G, parts, P.d_ja, lowest);
    ctx->launches++;
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    FGPU_CUDA_CHECK(ctx, cudaMemcpyAsync(h, lowest, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    FGPU_CUDA_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    int64_t low = P.nrows;                       // the lowest row of the parts after c
    int64_t end[kHostParts];
    for (int c = parts - 2; c >= 0; --c) {
        low = std::min<int64_t>(low, h[c + 1]);
        FGPU_CUDA_CHECK(ctx, cudaMemcpyAsync(&end[c], P.d_ia + low, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    }
    FGPU_CUDA_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c + 1 < parts; ++c) H.end[c] = end[c] & ~(int64_t)63;
    H.end[parts - 1] = P.nnz;
    H.count = parts;
    return FGPU_OK;
}

// Phase 2, then the values to the host (FP64 matrices): the slices run in parts, and the rows that no later part
// writes to leave meanwhile on a copy stream: with dofs numbered along the elements that is all but the last
// plane's. By the copy engine, or (FGPU_HOST_TRANSFER_DIRECT) by kernel stores into a page-locked, mapped buffer.
// Parts by the number of values: another part saves some of the gather's time and costs 5 to 10 us. Milliseconds
// with 1 / 2 / 4 / 8 / 12 parts through fgpu_assemble_matrix_host: P1 20^3 (0.13 M values) 0.037 / 0.046 / 0.065 / -,
// P2 14^3 (0.66 M) 0.070 / 0.067 / 0.075 / -, P2 20^3 (1.9 M) 0.124 / 0.126 / 0.128 / 0.135, P2 30^3 (6.3 M) 0.370 /
// 0.353 / 0.344 / 0.347, P2 64^3 (61 M, 2.55 ms on the link) 3.19 / 3.01 / 2.92 / 2.88 / 2.88, P3 40^3 (85 M) 4.32 /
// 4.09 / 3.96 / 3.90 / 3.89. On four copy streams in turn: P2 30^3 0.354, P2 20^3 0.134.
// Kernel stores: 32 blocks beside the gather (P2 30^3 0.359, 64 blocks 0.371; P2 64^3 2.94 and 2.92), on four streams
// in turn (on one, P2 64^3 3.07: a kernel's last stores run under the next one's), in one part up to 4 M values (P2
// 14^3 0.069, two parts 0.077; P2 30^3 0.367, four 0.359).
int host_parts(int64_t nnz, bool direct) {
    return nnz < ((int64_t)1 << (direct ? 22 : 19)) ? 1 : nnz < ((int64_t)1 << 22) ? 2 : nnz < ((int64_t)24 << 20) ? 4 : kHostParts;
}
constexpr int64_t kDirectBlocks = 32;
int launch_gather_phase_to_host(fgpu_ctx* ctx, fgpu_matrix* A, double* host) {
    const int64_t nnz = A->pattern->nnz;
    const bool direct = ctx->host_transfer == FGPU_HOST_TRANSFER_DIRECT;
    double* hdev = nullptr;
    if (direct) {
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, host) == cudaSuccess && pa.type == cudaMemoryTypeHost && pa.devicePointer)
            hdev = static_cast<double*>(pa.devicePointer);
        if (!hdev) {
            cudaGetLastError();
            ctx->err = "direct host transfer: the host buffer is not page-locked and mapped";
            return FGPU_ERR_INVALID;
        }
    }
    fgpu_space* V = A->space;
    const int parts = host_parts(nnz, direct);
    auto transfer = [&](int64_t k0, int64_t k1, cudaStream_t st, int64_t max_blocks) -> cudaError_t {
        if (!direct)
            return cudaMemcpyAsync(host + k0, (const double*)A->d_val + k0, (k1 - k0) * sizeof(double), cudaMemcpyDeviceToHost, st);
        const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((k1 - k0 + 255) / 256, max_blocks));
        values_to_host_kernel<<<(int)blocks, 256, 0, st>>>(k1 - k0, (const double*)A->d_val + k0, hdev + k0);
        ctx->launches++;
        return cudaGetLastError();
    };
    if (parts == 1) {                            // (the caller synchronises)
        const int rc = launch_gather_phase(ctx, A, 0);
        if (rc) return rc;
        FGPU_CUDA_CHECK(ctx, transfer(0, nnz, ctx->stream, (int64_t)sm_count(ctx) * 32));
        return FGPU_OK;
    }
    if (!ctx->copy_streams[0]) {
        for (int i = 0; i < 4; ++i) FGPU_CUDA_CHECK(ctx, cudaStreamCreateWithFlags(&ctx->copy_streams[i], cudaStreamNonBlocking));
        for (int i = 0; i < 5; ++i) FGPU_CUDA_CHECK(ctx, cudaEventCreateWithFlags(&ctx->copy_events[i], cudaEventDisableTiming));
    }
    const int rc = plan_parts(ctx, V, parts);
    if (rc) return rc;
    const GatherPlan& G = V->plan;
    const int64_t q = (G.nslices + parts - 1) / parts;
    PendingEvent ev;
    prof_begin(ctx, "assemble_gather", ev);
    int64_t done = 0;
    cudaError_t e = cudaSuccess;
    for (int c = 0; c < parts && e == cudaSuccess; ++c) {
        GatherPlan part = G;
        part.nslices = std::max<int64_t>(0, std::min(G.nslices, (c + 1) * q) - c * q);
        part.soff += c * q;
        part.pos0 += c * q * 32;
        part.pos1 += c * q * 32;
        if (part.nslices > 0) launch_slices<kModeDF64, false, false>(ctx, A, part, 256, 0, 4);
        if (c > 0) ctx->launches++;
        e = cudaGetLastError();
        const int64_t end = V->host_parts.end[c];
        if (end <= done || e != cudaSuccess) continue;
        const cudaStream_t cs = ctx->copy_streams[direct ? c & 3 : 0];
        // (the event is recorded again by the next part: a wait takes the record it finds)
        e = cudaEventRecord(ctx->copy_events[4], ctx->stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(cs, ctx->copy_events[4], 0);
        if (e == cudaSuccess) e = transfer(done, end, cs, kDirectBlocks);
        done = end;
    }
    prof_end(ctx, ev);
    // the context's stream waits for the copy streams: the caller's one wait covers all
    const int used = direct ? 4 : 1;
    for (int i = 0; i < used && e == cudaSuccess; ++i) {
        e = cudaEventRecord(ctx->copy_events[i], ctx->copy_streams[i]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, ctx->copy_events[i], 0);
    }
    if (e != cudaSuccess)
        for (int i = 0; i < used; ++i) cudaStreamSynchronize(ctx->copy_streams[i]);
    FGPU_CUDA_CHECK(ctx, e);
    return FGPU_OK;
}

int launch_batch_gather_slices(fgpu_ctx* ctx, int nprob, const BatchProblem* d_probs, const int64_t* d_slice_off, int64_t total_slices,
                               int f32, int threads, int accumulate) {
    const int blocks = (int)std::max<int64_t>(1, (total_slices + threads / 32 - 1) / (threads / 32));
    PendingEvent ev;
    prof_begin(ctx, "batch_gather", ev);
#define BATCH_GATHER(MODE, PIPE)                                                                                          \
    do {                                                                                                                  \
        if (accumulate) batch_gather_slices_kernel<MODE, PIPE, true><<<blocks, threads, 0, ctx->stream>>>(nprob, d_probs, d_slice_off, total_slices);  \
        else batch_gather_slices_kernel<MODE, PIPE, false><<<blocks, threads, 0, ctx->stream>>>(nprob, d_probs, d_slice_off, total_slices);            \
    } while (0)
    if (one_wave(ctx, total_slices)) {
        if (f32) BATCH_GATHER(kModeF32, true); else BATCH_GATHER(kModeDF64, true);
    } else {
        if (f32) BATCH_GATHER(kModeF32, false); else BATCH_GATHER(kModeDF64, false);
    }
#undef BATCH_GATHER
    prof_end(ctx, ev);
    FGPU_CUDA_CHECK(ctx, cudaGetLastError());
    return FGPU_OK;
}

}  // namespace fgpu

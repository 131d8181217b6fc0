// P1 and P2 Laplace/mass element matrices on affine tetrahedra in closed form, one lane per element.
//
// With exact quadrature the element matrix is a sum of few barycentric products: with
// h_ab = kappa |T| grad l_a . grad l_b, a P2 stiffness entry is (1/5) sum n h_ab with at most four terms
// and n in {3, -1, 8, 4} (p2_stiff_coef), a P1 entry is one h_ab, and the mass entries are small integers
// times mass |T| / 420 (P2) or / 20 (P1): about 1 300 double-float operations for the 55 entries of a P2
// element against 55 x 84 for the seven-term sums over the reference tensors. n and the mass integers are
// powers of two up to a factor 3, so the terms are exact multiples; a sum is compensated as everywhere
// (the high parts through TwoSum, errors and low parts in one binary32 accumulator, normalised once).
// Used where the form's quadrature rule integrates the products exactly (DevTables::closed).
#pragma once
#include <cstdint>
#include <type_traits>

#include "asm_device.cuh"
#include "entries.h"

namespace fgpu {

// compile-time loop: f(integral constant 0), ..., f(integral constant N - 1)
template <int I, int N, class F>
__device__ __forceinline__ void unrolled(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        unrolled<I + 1, N>(f);
    }
}

// numbers of the two modes and their compensated (plain) sums
struct ClosedDf {
    typedef df T;
    typedef float2 Out;
    struct Acc {
        float s, e;
    };
    static __device__ __forceinline__ T from(df x) { return x; }
    static __device__ __forceinline__ T scale(T x, float p2) { return df_scale(x, p2); }
    static __device__ __forceinline__ T triple(T x) {
        const float p = f_mul(3.0f, x.hi);
        return df{p, f_fma(3.0f, x.lo, f_fma(3.0f, x.hi, -p))};
    }
    static __device__ __forceinline__ Acc first(T x) { return Acc{x.hi, x.lo}; }
    static __device__ __forceinline__ void add(Acc& a, T x) {
        const df t = two_sum(a.s, x.hi);
        a.s = t.hi;
        a.e = f_add(a.e, f_add(t.lo, x.lo));
    }
    static __device__ __forceinline__ void scale_sum(Acc& a, float p2) {
        a.s = f_mul(a.s, p2);
        a.e = f_mul(a.e, p2);
    }
    static __device__ __forceinline__ Out out(Acc a) {
        const df r = quick_two_sum(a.s, a.e);
        return make_float2(r.hi, r.lo);
    }
};
struct ClosedF {
    typedef float T;
    typedef float Out;
    typedef float Acc;
    static __device__ __forceinline__ T from(df x) { return x.hi; }
    static __device__ __forceinline__ T scale(T x, float p2) { return f_mul(x, p2); }
    static __device__ __forceinline__ T triple(T x) { return f_mul(3.0f, x); }
    static __device__ __forceinline__ Acc first(T x) { return x; }
    static __device__ __forceinline__ void add(Acc& a, T x) { a = f_add(a, x); }
    static __device__ __forceinline__ void scale_sum(Acc& a, float p2) { a = f_mul(a, p2); }
    static __device__ __forceinline__ Out out(Acc a) { return a; }
};

__device__ __forceinline__ df df_over(df x, double inv) {
    const float h = (float)inv;
    return df_mul(x, df{h, (float)(inv - (double)h)});
}

// The factors that closed_entries expects in the record's stiffness and mass coefficients (given to
// geometry_df_record with kappa's and the mass's constant): h_ab (P2: / 5) is kappa J (B^T B)_ab / 4 times
// |T| / J, |T| = 4 J / 3 in the [-1, 1] reference element; the mass unit is mass |T| / 420 (P2) or / 20.
template <int N>
__device__ __forceinline__ df closed_stiff(df ksc) { return df_over(ksc, N == 10 ? 1.0 / 15.0 : 1.0 / 3.0); }
template <int N>
__device__ __forceinline__ df closed_mass(df mc) { return df_over(mc, N == 10 ? 1.0 / 315.0 : 1.0 / 15.0); }

// emit(t, value) for the entries t = 0 .. n (n + 1) / 2 - 1 of entry_order, t an integral constant;
// rec: the element's coefficient record with those factors
template <int MODE, int N, class F>
__device__ __forceinline__ void closed_entries(const float4* rec, F&& emit) {
    typedef typename std::conditional<MODE == kModeDF64, ClosedDf, ClosedF>::type P;
    typedef typename P::T T;
    float ch[7], cl[7];
    load_record_shared(rec, ch, cl, true);
    df h[10];
    h[sym4(1, 1)] = df{ch[0], cl[0]};
    h[sym4(2, 2)] = df{ch[1], cl[1]};
    h[sym4(3, 3)] = df{ch[2], cl[2]};
    h[sym4(1, 2)] = df{ch[3], cl[3]};
    h[sym4(1, 3)] = df{ch[4], cl[4]};
    h[sym4(2, 3)] = df{ch[5], cl[5]};
#pragma unroll
    for (int a = 1; a < 4; ++a) h[sym4(0, a)] = df_neg(df_add(df_add(h[sym4(1, a)], h[sym4(2, a)]), h[sym4(3, a)]));
    h[0] = df_neg(df_add(df_add(h[sym4(0, 1)], h[sym4(0, 2)]), h[sym4(0, 3)]));
    const T m = P::from(df{ch[6], cl[6]}), m3 = P::triple(m);
    T g[10], g3[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        g[k] = P::from(h[k]);
        if (N == 10) g3[k] = P::triple(g[k]);
    }
    unrolled<0, N*(N + 1) / 2>([&](auto I) {
        constexpr int t = decltype(I)::value;
        constexpr EntryOrder O = make_entry_order(4, N == 10 ? 2 : 1, N);
        constexpr int i = O.a[t], j = O.b[t];
        typename P::Acc acc;
        if constexpr (N == 4) {
            constexpr int k = sym4(i, j);
            acc = P::first(g[k]);
            P::add(acc, P::scale(m, i == j ? 2.0f : 1.0f));
        } else {
            // two edge functions: the sum over 4, scaled at the end
            constexpr float unit = i >= 4 && j >= 4 ? 4.0f : 1.0f;
            unrolled<0, bary_comps(i) * bary_comps(j)>([&](auto U) {
                constexpr int u = decltype(U)::value, k = u / bary_comps(j), l = u % bary_comps(j);
                if constexpr (i == j && k > l) return;       // equal to (l, k) of the same function: doubled there
                constexpr int n = p2_stiff_coef(i, k, j, l) * (i == j && k < l ? 2 : 1) / (int)unit;
                constexpr int gi = sym4(bary_comp(i, k), bary_comp(j, l));
                T x;
                if constexpr (n == 3) x = g3[gi];
                else if constexpr (n == 1) x = g[gi];
                else x = P::scale(g[gi], (float)n);
                if constexpr (u == 0) acc = P::first(x);
                else P::add(acc, x);
            });
            if constexpr (unit != 1.0f) P::scale_sum(acc, unit);
            constexpr int n = p2_mass_coef(i, j);
            if constexpr (n % 3 == 0) P::add(acc, P::scale(m3, (float)(n / 3)));
            else P::add(acc, P::scale(m, (float)n));
        }
        emit(I, P::out(acc));
    });
}

template <int MODE, int N>
constexpr int closed_stage_bytes() { return N * (N + 1) / 2 * 32 * (MODE == kModeDF64 ? 8 : 4); }

__device__ __forceinline__ void closed_stage_free() {     // the warp's stage may be written again
    if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
}

// one group of cnt <= 32 elements from e0 (in: the lane's element); stage: this warp's shared memory, whose
// earlier copy out runs on under the geometry
template <int MODE, int N>
__device__ __forceinline__ void closed_group(int64_t e0, int cnt, const GeoElem& in, const double* __restrict__ kappa, df kc, df mc,
                                             df ksc, unsigned char* stage, void* __restrict__ kbuf, int* __restrict__ status) {
    typedef typename std::conditional<MODE == kModeDF64, float2, float>::type V;
    constexpr int NTRI = N * (N + 1) / 2;
    const int lane = threadIdx.x & 31;
    V* st = reinterpret_cast<V*>(stage);
    V* out = reinterpret_cast<V*>(kbuf) + e0 * NTRI;
    float4 rec[4];
    if (lane < cnt) geometry_df_record<true>(in, kappa, kc, mc, ksc, rec, status);
    closed_stage_free();
    if (lane < cnt) {
        closed_entries<MODE, N>(rec, [&](auto I, V v) { st[lane * NTRI + decltype(I)::value] = v; });
    }
    if (cnt == 32) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out),
                         "r"((uint32_t)__cvta_generic_to_shared(stage)), "r"(closed_stage_bytes<MODE, N>())
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    } else {
        __syncwarp();
        for (int k = lane; k < cnt * NTRI; k += 32) out[k] = st[k];
    }
}
__device__ __forceinline__ void closed_stores_done() {
    if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace fgpu

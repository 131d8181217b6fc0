// Q2 hexahedra with trilinear geometry in double-float by sum factorisation.
//
// The basis and the M^3 Gauss points are tensor products, so the element matrix
//   K(i, j) = sum_q sum_rs G_rs(q) d_r phi_i(q) d_s phi_j(q) + m(q) phi_i(q) phi_j(q)
// is three one-dimensional contractions. With L and D the 1D functions and derivatives, for each (q2, q3)
//   A_11m = sum_q1 G_11 D_i1 D_j1 + m L_i1 L_j1,  A_12 = G_12 D_i1 L_j1,  A_13 = G_13 D_i1 L_j1,
//   A_22, A_23, A_33 = G_.. L_i1 L_j1,
// for each q3
//   LL = sum_q2 A_11m L_i2 L_j2 + A_22 D_i2 D_j2 + A_12(i, j) L_i2 D_j2 + A_12(j, i) D_i2 L_j2,
//   LD = sum_q2 A_13 L_i2 L_j2 + A_23 D_i2 L_j2,  DD = sum_q2 A_33 L_i2 L_j2,
// and K = sum_q3 LL L_i3 L_j3 + LD(i, j) L_i3 D_j3 + LD(j, i) D_i3 L_j3 + DD D_i3 D_j3: 9 200 products per
// element where entry by entry over the points takes 47 000 (27 points x 378 entries x 4, and W = G dphi).
// 128 threads take seven elements through each stage; a thread takes whole lines of products of 1D
// functions, whose factors are then compile-time constants (those that are zero at the middle point drop
// out) and whose operands are read from shared memory once. Seven elements: 126 pieces of A, 126 of LL and
// DD, 189 points and 189 pieces of LD, 315 pieces of K.
// Every sum is a compensated dot product (df_dot_term), rounded to double-float between the stages. The map's
// derivatives come from the seven mixed differences of the vertices, formed in binary64, so that no absolute
// coordinates cancel.
// Bound: FP32 issue (64 registers, 16 warps per SM by shared memory). Q2 31x32x33, 27 points: entry by entry
// with a warp per element 1050 us, here 180; error against binary64 4.8e-14 -> 8.2e-15.
#pragma once
#include "asm_device.cuh"
#include "closed.cuh"
#include "df64.h"

namespace fgpu {

constexpr int kHexBlock = 7;                                     // elements per block
constexpr int kHexA = 42, kHexB = 45 + 81 + 36;              // values per (q2, q3); per q3
template <int M>
constexpr int hex_q2_smem() {                                // points' coefficients, then LL / LD / DD; A, then K; geometry
    constexpr int g = 7 * M * M * M, b = kHexB * M, a = kHexA * M * M, k = 378;
    return kHexBlock * ((g > b ? g : b) + (a > k ? a : k) + 21) * 8;
}

namespace hexq2 {
constexpr double kS3 = 0.774596669241483377035853079956, kS2 = 0.577350269189625764509148780502;
template <int M>
constexpr double point(int q) { return M == 3 ? (q - 1) * kS3 : (2 * q - 1) * kS2; }
constexpr double L(int a, double t) { return a == 0 ? 0.5 * t * (t - 1.0) : a == 2 ? 0.5 * t * (t + 1.0) : (1.0 - t) * (1.0 + t); }
constexpr double D(int a, double t) { return a == 0 ? t - 0.5 : a == 2 ? t + 0.5 : -2.0 * t; }
enum { kLL, kDL, kLD, kDD };
template <int M>
constexpr double prod(int type, int q, int i, int j) {
    const double t = point<M>(q);
    return (type == kLL || type == kLD ? L(i, t) : D(i, t)) * (type == kLL || type == kDL ? L(j, t) : D(j, t));
}
constexpr int s6(int i, int j) { return i <= j ? i * 3 - i * (i - 1) / 2 + j - i : s6(j, i); }

// s + e += v * (the product of 1D functions of that type)
template <int M, int TYPE, int Q, int I, int J>
__device__ __forceinline__ void term(df v, float& s, float& e) {
    constexpr double c = prod<M>(TYPE, Q, I, J);
    if constexpr (c != 0.0) {
        constexpr float h = (float)c, l = (float)(c - (double)h);
        df_dot_term(v, df{h, l}, s, e);
    }
}
}  // namespace hexq2

template <int M>
__global__ void __launch_bounds__(128) hex_q2_kernel(int64_t nt, const double* __restrict__ xyz, const int32_t* __restrict__ hexes,
                                                     const float* __restrict__ qwh, const float* __restrict__ qwl,
                                                     const uint16_t* __restrict__ place, const double* __restrict__ d_kappa,
                                                     double kappa, double mass, const double* __restrict__ kscale,
                                                     float2* __restrict__ kbuf, int* __restrict__ status) {
    using namespace hexq2;
    constexpr int Q = M * M * M, NG = 7 * Q, NB = kHexB * M, NA = kHexA * M * M, NTRI = 378;
    constexpr int R1 = NG > NB ? NG : NB, R2 = NA > NTRI ? NA : NTRI;
    extern __shared__ __align__(16) float2 hex_smem[];
    float2* const r1 = hex_smem;                             // kHexBlock x R1: G (7 x Q), then LL 45, LD 81, DD 36 per q3
    float2* const r2 = hex_smem + kHexBlock * R1;                // A (kHexA x M M per element), then K (378 per element)
    float2* const geo = r2 + kHexBlock * R2;                     // kHexBlock x 21
    const int tid = threadIdx.x;
    const int64_t e0 = (int64_t)blockIdx.x * kHexBlock;
    const int ne = (int)(nt - e0 < kHexBlock ? nt - e0 : kHexBlock);
    auto get = [](float2 v) { return df{v.x, v.y}; };
    auto put = [](float2& o, float s, float e) {
        const df v = two_sum(s, e);
        o = make_float2(v.hi, v.lo);
    };
    // mixed differences of the vertices (a butterfly over the three signs), coordinate r of an element per thread
    if (tid < 3 * ne) {
        const int el = tid / 3, r = tid - 3 * el;
        const int32_t* t = hexes + 8 * (e0 + el);
        constexpr int kAt[8] = {0, 1, 3, 2, 4, 5, 7, 6};     // sign bits (x, y, z) of the vertices
        double d[8];
        const double x0 = xyz[3 * (int64_t)t[0] + r];
#pragma unroll
        for (int v = 0; v < 8; ++v) d[kAt[v]] = v == 0 ? 0.0 : xyz[3 * (int64_t)t[v] + r] - x0;
#pragma unroll
        for (int b = 1; b < 8; b <<= 1)
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (!(k & b)) {
                    const double lo = d[k], hi = d[k | b];
                    d[k] = hi + lo;
                    d[k | b] = hi - lo;
                }
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const df v = d2df(0.125 * d[k]);
            geo[el * 21 + (k - 1) * 3 + r] = make_float2(v.hi, v.lo);
        }
    }
    __syncthreads();
    // the points: G = w kappa / |det| C^T C (C: cofactors) and m = w |det| mass
    const df ksd = d2df(kscale ? *kscale : 1.0), massd = d2df(mass);
    for (int k = tid; k < ne * Q; k += 128) {
        const int el = k / Q, q = k - el * Q, q1 = q / (M * M), q2 = q / M % M, q3 = q % M;
        const float2* c = geo + el * 21;
        constexpr double s1 = M == 3 ? kS3 : kS2, s2 = M == 3 ? 0.6 : 1.0 / 3.0;
        constexpr float h1 = (float)s1, l1 = (float)(s1 - (double)h1), h2 = (float)s2, l2 = (float)(s2 - (double)h2);
        auto sign = [](int p) { return M == 3 ? (float)(p - 1) : (float)(2 * p - 1); };
        const float f1 = sign(q1), f2 = sign(q2), f3 = sign(q3);
        const df x = df_scale(df{h1, l1}, f1), y = df_scale(df{h1, l1}, f2), z = df_scale(df{h1, l1}, f3);
        const df yz = df_scale(df{h2, l2}, f2 * f3), xz = df_scale(df{h2, l2}, f1 * f3), xy = df_scale(df{h2, l2}, f1 * f2);
        df K[9];                                             // K[3 r + c]
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                // d / d xi_0: c_1 + c_3 eta + c_5 zeta + c_7 eta zeta, and so on
                const int i0 = d == 0 ? 1 : d == 1 ? 2 : 4, i1 = d == 2 ? 5 : 3, i2 = d == 0 ? 5 : 6;
                const df a = get(c[(i0 - 1) * 3 + r]);
                float s = a.hi, e = a.lo;
                df_dot_term(get(c[(i1 - 1) * 3 + r]), d == 0 ? y : x, s, e);
                df_dot_term(get(c[(i2 - 1) * 3 + r]), d == 2 ? y : z, s, e);
                df_dot_term(get(c[6 * 3 + r]), d == 0 ? yz : d == 1 ? xz : xy, s, e);
                K[3 * r + d] = two_sum(s, e);
            }
        df C[9];
        C[0] = df_sub(df_mul(K[4], K[8]), df_mul(K[5], K[7]));
        C[1] = df_sub(df_mul(K[5], K[6]), df_mul(K[3], K[8]));
        C[2] = df_sub(df_mul(K[3], K[7]), df_mul(K[4], K[6]));
        C[3] = df_sub(df_mul(K[2], K[7]), df_mul(K[1], K[8]));
        C[4] = df_sub(df_mul(K[0], K[8]), df_mul(K[2], K[6]));
        C[5] = df_sub(df_mul(K[1], K[6]), df_mul(K[0], K[7]));
        C[6] = df_sub(df_mul(K[1], K[5]), df_mul(K[2], K[4]));
        C[7] = df_sub(df_mul(K[2], K[3]), df_mul(K[0], K[5]));
        C[8] = df_sub(df_mul(K[0], K[4]), df_mul(K[1], K[3]));
        const df det = df_add(df_add(df_mul(K[0], C[0]), df_mul(K[1], C[1])), df_mul(K[2], C[2]));
        const df J = det.hi < 0.0f ? df_neg(det) : det;
        if (!(J.hi > 0.0f) || !isfinite(J.hi)) atomicOr(status, kStatusBadElement);
        const df w = df{__ldg(qwh + q), __ldg(qwl + q)};
        const df kap = df_mul(d2df(d_kappa ? d_kappa[e0 + el] : kappa), ksd);
        const df sc = df_mul(df_mul(w, kap), df_recip(J));
        float2* G = r1 + el * R1 + q;                        // 00, 11, 22, 01, 02, 12, m
        const int pa[6] = {0, 1, 2, 0, 0, 1}, pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            float s = 0.0f, e = 0.0f;
#pragma unroll
            for (int r = 0; r < 3; ++r) df_dot_term(C[3 * r + pa[t]], C[3 * r + pb[t]], s, e);
            const df g = df_mul(sc, two_sum(s, e));
            G[t * Q] = make_float2(g.hi, g.lo);
        }
        const df mm = df_mul(df_mul(w, J), massd);
        G[6 * Q] = make_float2(mm.hi, mm.lo);
    }
    __syncthreads();
    // A: a thread takes the sums over q1 at one (q2, q3), half of the types each
    // places: A_11m 0..5, A_22 6..11, A_23 12..17, A_33 18..23 (pairs s6), A_12 24..32, A_13 33..41 (pairs 3 i + j)
    for (int k = tid & 63; k < ne * M * M; k += 64) {
        const int el = k / (M * M), qq = k - el * M * M;
        const float2* G = r1 + el * R1 + qq;
        float2* A = r2 + el * R2 + qq;
        df g[M], h[M];
        auto load = [&](int t, df* o) {
#pragma unroll
            for (int q = 0; q < M; ++q) o[q] = get(G[t * Q + q * M * M]);
        };
        if (tid < 64) {
            load(0, g);
            load(6, h);
            unrolled<0, 9>([&](auto P) {
                constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
                if constexpr (i <= j) {
                    float s = 0.0f, e = 0.0f;
                    unrolled<0, M>([&](auto X) {
                        constexpr int q = decltype(X)::value;
                        term<M, kDD, q, i, j>(g[q], s, e);
                        term<M, kLL, q, i, j>(h[q], s, e);
                    });
                    put(A[s6(i, j) * M * M], s, e);
                }
            });
            load(3, g);
            unrolled<0, 9>([&](auto P) {
                constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
                float s = 0.0f, e = 0.0f;
                unrolled<0, M>([&](auto X) { term<M, kDL, decltype(X)::value, i, j>(g[decltype(X)::value], s, e); });
                put(A[(24 + 3 * i + j) * M * M], s, e);
            });
        } else {
            load(4, g);
            unrolled<0, 9>([&](auto P) {
                constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
                float s = 0.0f, e = 0.0f;
                unrolled<0, M>([&](auto X) { term<M, kDL, decltype(X)::value, i, j>(g[decltype(X)::value], s, e); });
                put(A[(33 + 3 * i + j) * M * M], s, e);
            });
#pragma unroll 1
            for (int t = 0; t < 3; ++t) {                    // G_11, G_12, G_22
                load(t == 0 ? 1 : t == 1 ? 5 : 2, g);
                unrolled<0, 9>([&](auto P) {
                    constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
                    if constexpr (i <= j) {
                        float s = 0.0f, e = 0.0f;
                        unrolled<0, M>([&](auto X) { term<M, kLL, decltype(X)::value, i, j>(g[decltype(X)::value], s, e); });
                        put(A[(6 + 6 * t + s6(i, j)) * M * M], s, e);
                    }
                });
            }
        }
    }
    __syncthreads();
    // LL and DD: a thread takes one q3 and one pair i1 <= j1
    for (int k = tid; k < ne * 6 * M; k += 128) {
        const int el = k / (6 * M), u = k - el * 6 * M, p1 = u / M, q3 = u - p1 * M;
        const int i1 = p1 < 3 ? 0 : p1 < 5 ? 1 : 2, j1 = p1 < 3 ? p1 : p1 < 5 ? p1 - 2 : 2;
        const float2* A = r2 + el * R2 + q3;
        float2* B = r1 + el * R1 + q3 * kHexB;
        df a[M], b[M], c[M], d[M];
#pragma unroll
        for (int q = 0; q < M; ++q) {
            a[q] = get(A[p1 * M * M + q * M]);
            b[q] = get(A[(6 + p1) * M * M + q * M]);
            c[q] = get(A[(24 + 3 * i1 + j1) * M * M + q * M]);
            d[q] = get(A[(24 + 3 * j1 + i1) * M * M + q * M]);
        }
        unrolled<0, 9>([&](auto P) {
            constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
            if (i1 == j1 && i > j) return;
            float s = 0.0f, e = 0.0f;
            unrolled<0, M>([&](auto X) {
                constexpr int q = decltype(X)::value;
                term<M, kLL, q, i, j>(a[q], s, e);
                term<M, kDD, q, i, j>(b[q], s, e);
                term<M, kLD, q, i, j>(c[q], s, e);
                term<M, kDL, q, i, j>(d[q], s, e);
            });
            const int x = 3 * i1 + i, y = 3 * j1 + j;        // x <= y
            put(B[9 * x - x * (x - 1) / 2 + y - x], s, e);
        });
#pragma unroll
        for (int q = 0; q < M; ++q) a[q] = get(A[(18 + p1) * M * M + q * M]);
        unrolled<0, 9>([&](auto P) {
            constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
            if constexpr (i <= j) {
                float s = 0.0f, e = 0.0f;
                unrolled<0, M>([&](auto X) { term<M, kLL, decltype(X)::value, i, j>(a[decltype(X)::value], s, e); });
                put(B[126 + p1 * 6 + s6(i, j)], s, e);
            }
        });
    }
    // LD: one q3 and one pair (i1, j1)
    for (int k = tid; k < ne * 9 * M; k += 128) {
        const int el = k / (9 * M), u = k - el * 9 * M, p1 = u / M, q3 = u - p1 * M, i1 = p1 / 3, j1 = p1 - 3 * i1;
        const float2* A = r2 + el * R2 + q3;
        float2* B = r1 + el * R1 + q3 * kHexB + 45 + 27 * i1 + 3 * j1;
        df a[M], b[M];
#pragma unroll
        for (int q = 0; q < M; ++q) {
            a[q] = get(A[(33 + p1) * M * M + q * M]);
            b[q] = get(A[(12 + s6(i1, j1)) * M * M + q * M]);
        }
        unrolled<0, 9>([&](auto P) {
            constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
            float s = 0.0f, e = 0.0f;
            unrolled<0, M>([&](auto X) {
                constexpr int q = decltype(X)::value;
                term<M, kLL, q, i, j>(a[q], s, e);
                term<M, kDL, q, i, j>(b[q], s, e);
            });
            put(B[9 * i + j], s, e);
        });
    }
    __syncthreads();
    // K: a thread takes one pair x = (i1, i2) <= y = (j1, j2)
    for (int k = tid; k < ne * 45; k += 128) {
        const int el = k / 45;
        int y = k - el * 45, x = 0;
#pragma unroll
        for (int r = 9; r > 1; --r)
            if (y >= r && x == 9 - r) {
                y -= r;
                ++x;
            }
        const int p = k - el * 45;
        y += x;
        const float2* B = r1 + el * R1;
        const int dd = 126 + 6 * s6(x / 3, y / 3) + s6(x % 3, y % 3);
        df a[M], b[M], c[M], d[M];
#pragma unroll
        for (int q = 0; q < M; ++q) {
            a[q] = get(B[q * kHexB + p]);
            b[q] = get(B[q * kHexB + 45 + 9 * x + y]);
            c[q] = get(B[q * kHexB + 45 + 9 * y + x]);
            d[q] = get(B[q * kHexB + dd]);
        }
        float2* K = r2 + el * NTRI;
        const uint16_t* at = place + 81 * x + 3 * y;
        unrolled<0, 9>([&](auto P) {
            constexpr int i = decltype(P)::value / 3, j = decltype(P)::value % 3;
            if (x == y && i > j) return;
            float s = 0.0f, e = 0.0f;
            unrolled<0, M>([&](auto X) {
                constexpr int q = decltype(X)::value;
                term<M, kLL, q, i, j>(a[q], s, e);
                term<M, kLD, q, i, j>(b[q], s, e);
                term<M, kDL, q, i, j>(c[q], s, e);
                term<M, kDD, q, i, j>(d[q], s, e);
            });
            put(K[__ldg(at + 27 * i + j)], s, e);
        });
    }
    __syncthreads();
    for (int k = tid; k < ne * NTRI; k += 128) kbuf[e0 * NTRI + k] = r2[k];
}

}  // namespace fgpu

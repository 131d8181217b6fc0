// Order of an element's upper-triangle entries in the two-phase element buffer: grouped by the smallest
// vertex, edge, face or cell that holds both dofs, small ones first, row-major inside a group. Usable at
// compile time (kernels with one lane per element address their accumulators by it) and on the host.
#pragma once
#include <cstdint>

namespace fgpu {

// vertices of the cells' edges and faces (the local order of kEdgeVerts, kFaceVerts, kHexEdgeVerts, kHexFaceVerts)
constexpr int kTetE[6][2] = {{1, 2}, {2, 0}, {0, 1}, {0, 3}, {1, 3}, {2, 3}};
constexpr int kTetF[4][3] = {{1, 2, 3}, {0, 2, 3}, {0, 1, 3}, {0, 1, 2}};
constexpr int kHexE[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {1, 5}, {5, 4}, {4, 0}, {2, 6}, {6, 5}, {3, 7}, {7, 6}, {4, 7}};
constexpr int kHexF[6][4] = {{0, 1, 2, 3}, {0, 1, 5, 4}, {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 0, 4, 7}, {4, 5, 6, 7}};

// the vertices that a local dof's entity spans, as a bit mask
constexpr uint32_t dof_span(int cell_vertices, int order, int dof) {
    if (dof < cell_vertices) return 1u << dof;
    dof -= cell_vertices;
    uint32_t m = 0;
    if (cell_vertices == 8) {
        if (dof < 12) return (1u << kHexE[dof][0]) | (1u << kHexE[dof][1]);
        if (dof < 18) {
            for (int k = 0; k < 4; ++k) m |= 1u << kHexF[dof - 12][k];
            return m;
        }
        return 0xFFu;
    }
    const int per_edge = order - 1;
    if (dof < 6 * per_edge) return (1u << kTetE[dof / per_edge][0]) | (1u << kTetE[dof / per_edge][1]);
    for (int k = 0; k < 3; ++k) m |= 1u << kTetF[dof - 6 * per_edge][k];
    return m;
}

struct EntryOrder {
    int n = 0, ntri = 0;
    uint8_t a[378] = {}, b[378] = {};      // the pair a <= b of entry t
    int16_t at[27][27] = {};               // (a, b) in either order -> t
};

constexpr EntryOrder make_entry_order(int cell_vertices, int order, int n) {
    EntryOrder E;
    E.n = n;
    uint32_t holder[27] = {};
    int nh = 0;
    for (int v = 0; v < cell_vertices; ++v) holder[nh++] = 1u << v;
    if (cell_vertices == 8) {
        for (int k = 0; k < 12; ++k) holder[nh++] = (1u << kHexE[k][0]) | (1u << kHexE[k][1]);
        for (int k = 0; k < 6; ++k) holder[nh++] = (1u << kHexF[k][0]) | (1u << kHexF[k][1]) | (1u << kHexF[k][2]) | (1u << kHexF[k][3]);
    } else {
        for (int k = 0; k < 6; ++k) holder[nh++] = (1u << kTetE[k][0]) | (1u << kTetE[k][1]);
        for (int k = 0; k < 4; ++k) holder[nh++] = (1u << kTetF[k][0]) | (1u << kTetF[k][1]) | (1u << kTetF[k][2]);
    }
    holder[nh++] = (1u << cell_vertices) - 1u;
    for (int g = 0; g < nh; ++g)
        for (int a = 0; a < n; ++a)
            for (int b = a; b < n; ++b) {
                const uint32_t m = dof_span(cell_vertices, order, a) | dof_span(cell_vertices, order, b);
                int first = 0;
                while ((holder[first] & m) != m) ++first;
                if (first != g) continue;
                E.a[E.ntri] = (uint8_t)a;
                E.b[E.ntri] = (uint8_t)b;
                E.at[a][b] = E.at[b][a] = (int16_t)E.ntri;
                ++E.ntri;
            }
    return E;
}

// ---- P1 and P2 tetrahedra in barycentric coordinates ----
// A vertex function of P2 has one barycentric derivative, (4 l_i - 1) along i; an edge function 4 l_p l_q
// has two, 4 l_q along p and 4 l_p along q. Pairs (a, b) of the four coordinates are kept as a <= b.
constexpr int sym4(int a, int b) { return a <= b ? a * 4 - a * (a - 1) / 2 + b - a : sym4(b, a); }
constexpr int bary_comps(int i) { return i < 4 ? 1 : 2; }
constexpr int bary_comp(int i, int k) { return i < 4 ? i : kTetE[i - 4][k]; }        // the coordinate of derivative k
constexpr int bary_factor(int i, int k) { return i < 4 ? i : kTetE[i - 4][1 - k]; }  // the l in it

// 5 / |T| times the integral of derivative k of function i times derivative m of function j over T (P2):
// 3 or -1 for two vertex functions or a vertex and an edge function, 8 or 4 for two edge functions
constexpr int p2_stiff_coef(int i, int k, int j, int m) {
    const bool same = bary_factor(i, k) == bary_factor(j, m);
    return i >= 4 && j >= 4 ? (same ? 8 : 4) : (same ? 3 : -1);
}
// 420 / |T| times the integral of phi_i phi_j (P2)
constexpr int p2_mass_coef(int i, int j) {
    if (i < 4 && j < 4) return i == j ? 6 : 1;
    if (i < 4 || j < 4) {
        const int v = i < 4 ? i : j, e = (i < 4 ? j : i) - 4;
        return kTetE[e][0] == v || kTetE[e][1] == v ? -4 : -6;
    }
    if (i == j) return 32;
    const int a = kTetE[i - 4][0], b = kTetE[i - 4][1], c = kTetE[j - 4][0], d = kTetE[j - 4][1];
    return a == c || a == d || b == c || b == d ? 16 : 8;
}

}  // namespace fgpu

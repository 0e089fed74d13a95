// straight.cuh -- element arithmetic of straight-sided tetrahedra (new).
//
// A TET10 whose mid-edge nodes sit at the edge midpoints (every TET4, every mesh of
// TetGen or of the structured mesher before it is curved) has one Jacobian for all
// quadrature points, so its geometry is 10 values -- J^-1 and det J -- instead of 10 per
// point, and the displacement gradient is linear in the barycentric coordinates: its
// values at the four vertices give it at every point.  For the linear operator (the SVK
// tangent at F = I) the sums over the points of a symmetric rule collapse too:
//   sum_q w_q L_i(q) sigma(q) = (m_d - m_o) sigma_i + m_o sum_j sigma_j,
// m_d = sum_q w_q L_i^2, m_o = sum_q w_q L_i L_j, so K p of an element is four vertex
// stresses and ten nodal forces: about 490 FP64 operations against about 1,500 point by
// point, and 80 bytes of geometry against 400.
//
// calc_dndu_pre decides whether a mesh qualifies (Tiling::straight): every mid-edge node
// within 4 units in the last place of its edge's midpoint (the rounding of the
// coordinates themselves, which every evaluation of J carries), no degenerate element,
// and for TET10 a rule of the Keast form (centroid plus the four permutations of
// (a, b, b, b), equal weights).  Everything else keeps the per-point streams.
#pragma once

#include "element.cuh"

namespace tlfea {

// Edge of TET10 node 4 + k.
__host__ __device__ constexpr int edge_i(int k) { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 0 : k == 3 ? 0 : k == 4 ? 1 : 2; }
__host__ __device__ constexpr int edge_j(int k) { return k == 0 ? 1 : k == 1 ? 2 : k == 2 ? 2 : 3; }
// Mid-edge node of corners i != j.
__host__ __device__ constexpr int edge_node(int i, int j) {
    return (i + j == 1) ? 4 : (i + j == 2) ? 6 : (i + j == 3) ? ((i == 0 || j == 0) ? 7 : 5) : (i + j == 4) ? 8 : 9;
}

// The rule's moments, per unit det J: c1 = 4 (m_d - m_o), c2 = 4 m_o, c3 = sum_q w_q L_j
// (the same for every j); TET4: c1 = the weight.
struct LinRule {
    double c1, c2, c3;
};

// Symmetric index of (i, j): 0 xx, 1 yy, 2 zz, 3 xy, 4 xz, 5 yz.
__host__ __device__ constexpr int sym_ij(int i, int j) { return i == j ? i : (i + j == 1 ? 3 : (i + j == 2 ? 4 : 5)); }

// dx/dxi at the four vertices (TET10) or the one point (TET4) for one component, from the
// node values relative to the first node.
template <typename R, int NPE>
__device__ __forceinline__ void vertex_gradients(const R (&d)[NPE], R (&G)[NPE == 10 ? 4 : 1][3]) {
    if constexpr (NPE == 10) {
        const R e1 = R(4) * d[4], e2 = R(4) * d[6], e3 = R(4) * d[7];
        const R m12 = R(4) * d[5], m13 = R(4) * d[8], m23 = R(4) * d[9];
        G[0][0] = e1 - d[1];
        G[0][1] = e2 - d[2];
        G[0][2] = e3 - d[3];
        G[1][0] = R(3) * d[1] - e1;
        G[1][1] = m12 - d[2] - e1;
        G[1][2] = m13 - d[3] - e1;
        G[2][0] = m12 - d[1] - e2;
        G[2][1] = R(3) * d[2] - e2;
        G[2][2] = m23 - d[3] - e2;
        G[3][0] = m13 - d[1] - e3;
        G[3][1] = m23 - d[2] - e3;
        G[3][2] = R(3) * d[3] - e3;
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) G[0][k] = d[k + 1];
    }
}

// Element forces of the linear operator, fe[(3a + c) * TILE_ELEMS] = (K p)_a,c, from p at
// the element's nodes (p(a, c)), taken relative to the first node: the operator drops the
// common part of p, and so does its rounding.  One component of p at a time, so that nine
// differences and the vertex stresses are the only long-lived registers.
template <typename R, int NPE, typename P>
__device__ __forceinline__ void lin_element(const R (&ji)[9], R det, R lam, R mu, const LinRule& rule, P p, R* fe) {
    constexpr int TE = TILE_ELEMS;
    constexpr int NV = NPE == 10 ? 4 : 1;  // points at which the stress is formed
    R s[NV][6];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const auto p0 = p(0, c);
        R G[NV][3];
        R d[NPE];
        d[0] = R(0);
#pragma unroll
        for (int a = 1; a < NPE; ++a) d[a] = R(p(a, c) - p0);
        vertex_gradients<R, NPE>(d, G);
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const R h = G[v][0] * ji[j] + G[v][1] * ji[3 + j] + G[v][2] * ji[6 + j];
                const int k = sym_ij(c, j);
                if (c <= j)
                    s[v][k] = h;  // xx, then xy and xz; yy, yz; zz
                else
                    s[v][k] += h;
            }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const R lt = lam * (s[v][0] + s[v][1] + s[v][2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s[v][k] = R(2) * mu * s[v][k] + lt;
            s[v][3 + k] *= mu;
        }
    }
    R gl[4][3];  // dL_k/dx
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        gl[1][j] = ji[j];
        gl[2][j] = ji[3 + j];
        gl[3][j] = ji[6 + j];
        gl[0][j] = -(ji[j] + ji[3 + j] + ji[6 + j]);
    }
    if constexpr (NPE == 10) {
        const R c1 = R(rule.c1) * det, c2 = R(rule.c2) * det, c3 = R(rule.c3) * det;
        R sb[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const R t = (s[0][k] + s[1][k]) + (s[2][k] + s[3][k]);
            sb[k] = c3 * t;
#pragma unroll
            for (int v = 0; v < 4; ++v) s[v][k] = c1 * s[v][k] + c2 * t;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int i = edge_i(k), j = edge_j(k);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                R f = R(0);
#pragma unroll
                for (int m = 0; m < 3; ++m) f += s[i][sym_ij(c, m)] * gl[j][m] + s[j][sym_ij(c, m)] * gl[i][m];
                fe[((4 + k) * 3 + c) * TE] = f;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                R f = R(0);
#pragma unroll
                for (int m = 0; m < 3; ++m) f += (s[i][sym_ij(c, m)] - sb[sym_ij(c, m)]) * gl[i][m];
                fe[(i * 3 + c) * TE] = f;
            }
    } else {
        const R w = R(rule.c1) * det;
#pragma unroll
        for (int k = 0; k < 6; ++k) s[0][k] *= w;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                fe[(i * 3 + c) * TE] =
                    s[0][sym_ij(c, 0)] * gl[i][0] + s[0][sym_ij(c, 1)] * gl[i][1] + s[0][sym_ij(c, 2)] * gl[i][2];
    }
}

// Node values in global memory as 32-byte records (x, y, z, unused): one 256-bit access and
// one sector per node, where 24-byte records take three accesses and straddle sectors.
__device__ __forceinline__ void ld_node(const double* p, double v[3]) {
    [[maybe_unused]] double w;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(w) : "l"(p));
}
// The same past L1, for values that other blocks of a running kernel write.
__device__ __forceinline__ void ld_node_shared(const double* p, double v[3]) {
    [[maybe_unused]] double w;
    asm volatile("ld.relaxed.gpu.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_node(double* p, double a, double b, double c) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(0.0) : "memory");
}

// Sum of the tile's element forces at one node: entries [beg, end) of its incidence list, in
// that order, NK = 6 loads in flight at a time (a corner node has up to 24).
template <typename R>
__device__ __forceinline__ void tile_node_sum(const R* fe, const uint16_t* incs, int beg, int end, double& s0,
                                              double& s1, double& s2) {
    constexpr int TE = TILE_ELEMS, NK = 6;
    s0 = s1 = s2 = 0.0;
    for (int k = beg; k < end; k += NK) {
        R v[NK][3];
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            const int ent = incs[min(k + j, end - 1)];
            const int base = (ent >> TILE_SHIFT) * 3 * TE + (ent & (TE - 1));
#pragma unroll
            for (int d = 0; d < 3; ++d) v[j][d] = (k + j < end) ? fe[base + d * TE] : R(0);
        }
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            s0 += v[j][0];
            s1 += v[j][1];
            s2 += v[j][2];
        }
    }
}

// Opt a tile kernel into the largest dynamic shared memory (the same value whatever the
// mesh, so meshes and threads cannot undercut one another).
constexpr size_t STRAIGHT_MAX_SMEM = 226 * 1024;
inline cudaError_t allow_tile_smem(const void* kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STRAIGHT_MAX_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    return e;
}

// Moments of the element's rule (valid where the tiling is straight).
inline LinRule lin_rule(const tlfea_element_s* h) {
    LinRule r{h->qw[0], 0.0, 0.0};
    if (h->npe != 10) return r;
    const double w0 = h->qw[0], w1 = h->qw[1];
    const double a = 1.0 - h->qx[1] - h->qy[1] - h->qz[1], b = h->qx[1];  // point 1: L = (a, b, b, b)
    const double md = w0 / 16.0 + w1 * (a * a + 3.0 * b * b);
    const double mo = w0 / 16.0 + w1 * (2.0 * a * b + 2.0 * b * b);
    r.c1 = 4.0 * (md - mo);
    r.c2 = 4.0 * mo;
    r.c3 = w0 / 4.0 + w1 * (a + 3.0 * b);
    return r;
}

// Whether the element's rule has the form the straight-sided arithmetic assumes: for TET4 any
// point will do (svk_element takes its mass from the point itself).
inline bool rule_is_symmetric(const tlfea_element_s* h) {
    if (h->npe != 10) return true;
    const double tol = 4e-16;
    const QpBary q = qp_bary(h);
    const double a = q.L[1][0], b = q.L[1][1];
    for (int p = 0; p < 5; ++p)
        for (int i = 0; i < 4; ++i) {
            const double want = p == 0 ? 0.25 : (i == p - 1 ? a : b);
            if (!(q.L[p][i] - want <= tol && want - q.L[p][i] <= tol)) return false;
        }
    for (int p = 2; p < 5; ++p)
        if (!(h->qw[p] - h->qw[1] <= tol && h->qw[1] - h->qw[p] <= tol)) return false;
    return true;
}

}  // namespace tlfea

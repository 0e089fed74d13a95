// straight_svk.cuh -- the nonlinear (SVK) element force of straight-sided tetrahedra; see
// straight.cuh for which meshes qualify and why their geometry is one Jacobian.
#pragma once

#include "straight.cuh"

namespace tlfea {

// The rule and its mass moments for the nonlinear element: point 0 the centroid (weight w0),
// points 1..4 L = (a, b, b, b) and its permutations (weight w1); TET4: w0 and L its one point,
// anywhere (the force does not depend on it, the mass does).
// TET10's mass moments m = sum_q w_q N_a N_b, per unit rho det J, of the pairs (vertex, itself),
// (vertex, other vertex), (vertex, its edge), (vertex, edge not at it), (edge, itself),
// (edge, edge sharing a vertex), (edge, opposite edge).
struct SvkRule {
    double a, b, w0, w1;
    double vv, vw, ve, vf, ee, ea, eo;
    double L[4];
};

// Rows of F (FP64, from positions) or H = F - I (FP32, from displacements) at the vertices:
// V[v][c][:] = (dx_c/dxi at v) J^-1.
template <typename R, int NPE, typename X>
__device__ __forceinline__ void vertex_f(const R (&ji)[9], X x, R (&V)[NPE == 10 ? 4 : 1][3][3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        // FP64 up to the vertex gradients: their coefficients of 3 and 4 would amplify FP32 rounding
        const double x0 = x(0, c);
        double d[NPE], G[NPE == 10 ? 4 : 1][3];
        d[0] = 0.0;
#pragma unroll
        for (int a = 1; a < NPE; ++a) d[a] = x(a, c) - x0;
        vertex_gradients<double, NPE>(d, G);
#pragma unroll
        for (int v = 0; v < (NPE == 10 ? 4 : 1); ++v)
#pragma unroll
            for (int j = 0; j < 3; ++j) V[v][c][j] = R(G[v][0]) * ji[j] + R(G[v][1]) * ji[3 + j] + R(G[v][2]) * ji[6 + j];
    }
}

// P = F S, S = lambda tr(E) I + 2 mu E, E = (F^T F - I) / 2 (the SVK law, SVK.cuh:17-39), with
// F given (FP64) or H = F - I (FP32: E = (H + H^T + H^T H) / 2, no cancellation); with DAMP
// the Kelvin-Voigt part S += 2 eta Ed + lamd tr(Ed) I, Ed = (Fd^T F + F^T Fd) / 2.
template <typename R, bool DAMP>
__device__ __forceinline__ void svk_p(const R (&F)[3][3], const R (&Fd)[3][3], R lam, R mu, R eta, R lamd,
                                      R (&P)[3][3]) {
    constexpr int SI[6] = {0, 1, 2, 0, 0, 1}, SJ[6] = {0, 1, 2, 1, 2, 2};
    constexpr bool DISP = sizeof(R) == 4;
    R M[6], S[6];  // M = 2 E
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int i = SI[k], j = SJ[k];
        R m = DISP ? F[i][j] + F[j][i] : (i == j ? R(-1) : R(0));
#pragma unroll
        for (int c = 0; c < 3; ++c) m += F[c][i] * F[c][j];
        M[k] = m;
    }
    R t = R(0.5) * lam * (M[0] + M[1] + M[2]);
    if constexpr (DAMP) {
        R D[6];  // 2 Ed
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int i = SI[k], j = SJ[k];
            R m = DISP ? Fd[i][j] + Fd[j][i] : R(0);
#pragma unroll
            for (int c = 0; c < 3; ++c) m += Fd[c][i] * F[c][j] + F[c][i] * Fd[c][j];
            D[k] = m;
        }
        t += R(0.5) * lamd * (D[0] + D[1] + D[2]);
#pragma unroll
        for (int k = 0; k < 6; ++k) S[k] = mu * M[k] + eta * D[k];
    } else {
#pragma unroll
        for (int k = 0; k < 6; ++k) S[k] = mu * M[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) S[k] += t;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            R v = DISP ? S[sym_ij(i, j)] : R(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) v += F[i][k] * S[sym_ij(k, j)];
            P[i][j] = v;
        }
}

// Element forces of the SVK law, fe[(3a + c) * TILE_ELEMS], at the node values x(a, c)
// (positions in FP64, displacements in FP32 mode); v(a, c): velocities (DAMP); w(a, c): with
// MASS the values rho (v - v_prev) / dt whose consistent-mass product is added.  F is linear in
// the element, so its four vertex values give it at the five points; the points' P collapse
// into four vertex moments the same way.  About 800 FP64 operations a TET10 (1,020 with MASS),
// against 1,550 (2,050) point by point.
// FP32: the points' P enter the moments by their differences to the centroid's.  The corners'
// moments drop the common part, which is most of P in a smooth field, and in FP32 its rounding
// would stay behind.  60 Nesterov iterations, distance from 64 bits over the per-point kernels':
// 233,280 elements 1.27 without the differences, 0.5 to 0.8 with them; 1,920 elements 1.0 to 1.25
// and 0.83 to 0.87; the largest found, 15,360 elements under an axial load with a short step, 1.42
// and 1.10.
template <typename R, int NPE, bool DAMP, bool MASS, typename X, typename V, typename W>
__device__ __forceinline__ void svk_element(const R (&ji)[9], R det, R lam, R mu, R eta, R lamd, const SvkRule& rule,
                                            X x, V v, W w, R* fe) {
    constexpr int TE = TILE_ELEMS;
    constexpr int NV = NPE == 10 ? 4 : 1;
    R B[NV][3][3], Bd[DAMP ? NV : 1][3][3];
    vertex_f<R, NPE>(ji, x, B);
    if constexpr (DAMP) vertex_f<R, NPE>(ji, v, Bd);
    R sb[3][3];
    if constexpr (NPE == 10) {
        const R ra = R(rule.a - rule.b), rb = R(rule.b);
        R sum[3][3], sumd[3][3], F[3][3], Fd[3][3], P[3][3], T[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                sum[i][j] = (B[0][i][j] + B[1][i][j]) + (B[2][i][j] + B[3][i][j]);
                F[i][j] = R(0.25) * sum[i][j];
                sum[i][j] *= rb;
                if constexpr (DAMP) {
                    sumd[i][j] = (Bd[0][i][j] + Bd[1][i][j]) + (Bd[2][i][j] + Bd[3][i][j]);
                    Fd[i][j] = R(0.25) * sumd[i][j];
                    sumd[i][j] *= rb;
                }
            }
        svk_p<R, DAMP>(F, Fd, lam, mu, eta, lamd, P);
        constexpr bool DIFF = sizeof(R) == 4;
        const R a0 = R(DIFF ? rule.w0 + 4.0 * rule.w1 : rule.w0) * det, a1 = R(rule.w1) * det;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                T[i][j] = R(0);
                sb[i][j] = DIFF ? P[i][j] : a0 * P[i][j];
            }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    F[i][j] = sum[i][j] + ra * B[q][i][j];
                    if constexpr (DAMP) Fd[i][j] = sumd[i][j] + ra * Bd[q][i][j];
                }
            svk_p<R, DAMP>(F, Fd, lam, mu, eta, lamd, P);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    if constexpr (DIFF) P[i][j] -= sb[i][j];
                    T[i][j] += P[i][j];
                    B[q][i][j] = P[i][j];
                }
        }
        // sb = sum_q w_q P_q det J; B_v = sum_q w_q (4 L_v - 1) P_q det J, which the centroid is
        // not part of (formed as 4 sum_q w_q L_v P_q - sb it cancels), nor a part common to the points
        const R d1 = R(4) * a1 * ra, d2 = R(rule.w1 * (4.0 * rule.b - 1.0)) * det;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                sb[i][j] = (DIFF ? a0 * sb[i][j] : sb[i][j]) + a1 * T[i][j];
                T[i][j] *= d2;
#pragma unroll
                for (int q = 0; q < 4; ++q) B[q][i][j] = T[i][j] + d1 * B[q][i][j];
            }
    } else {
        svk_p<R, DAMP>(B[0], Bd[0], lam, mu, eta, lamd, sb);
        const R a0 = R(rule.w0) * det;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) sb[i][j] *= a0;
    }
    R gl[4][3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        gl[1][j] = ji[j];
        gl[2][j] = ji[3 + j];
        gl[3][j] = ji[6 + j];
        gl[0][j] = -(ji[j] + ji[3 + j] + ji[6 + j]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        R f[NPE];
        if constexpr (MASS) {
            R m[NPE], sv = R(0);
            if constexpr (NPE == 10) {
                R adj[4], se = R(0);
#pragma unroll
                for (int a = 0; a < NPE; ++a) m[a] = R(w(a, c));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sv += m[i];
                    adj[i] = R(0);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j != i) adj[i] += m[edge_node(i, j)];
                    se += adj[i];
                }
                se *= R(0.5);  // every edge counted at both ends
                const R vv = R(rule.vv - rule.vw) * det, vw = R(rule.vw) * det;
                const R ve = R(rule.ve - rule.vf) * det, vf = R(rule.vf) * det;
                const R ee = R(rule.ee - rule.ea) * det, ea = R(rule.ea) * det, eo = R(rule.eo - rule.ea) * det;
                const R base_v = vw * sv + vf * se, base_e = vf * sv + ea * se;
#pragma unroll
                for (int i = 0; i < 4; ++i) f[i] = base_v + vv * m[i] + ve * adj[i];
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int i = edge_i(k), j = edge_j(k);
                    const int o = edge_node(i == 0 ? (j == 1 ? 2 : 1) : 0,
                                            i == 0 ? (j == 3 ? 2 : 3) : (i + j == 3 ? 3 : (i + j == 4 ? 2 : 1)));
                    f[4 + k] = base_e + ve * (m[i] + m[j]) + ee * m[4 + k] + eo * m[o];
                }
            } else {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    m[a] = R(w(a, c));
                    sv += R(rule.L[a]) * m[a];
                }
                sv *= R(rule.w0) * det;
#pragma unroll
                for (int a = 0; a < 4; ++a) f[a] = R(rule.L[a]) * sv;
            }
        } else {
#pragma unroll
            for (int a = 0; a < NPE; ++a) f[a] = R(0);
        }
        if constexpr (NPE == 10) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    f[i] += B[i][c][m] * gl[i][m];
                    B[i][c][m] += sb[c][m];  // 4 sum_q w_q L_v P_q det J
                }
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const int i = edge_i(k), j = edge_j(k);
#pragma unroll
                for (int m = 0; m < 3; ++m) f[4 + k] += B[i][c][m] * gl[j][m] + B[j][c][m] * gl[i][m];
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int m = 0; m < 3; ++m) f[i] += sb[c][m] * gl[i][m];
        }
#pragma unroll
        for (int a = 0; a < NPE; ++a) fe[(a * 3 + c) * TE] = f[a];
    }
}

// The constants of svk_element (valid where the tiling is straight).
inline SvkRule svk_rule(const tlfea_element_s* h) {
    SvkRule r{};
    const QpBary q = qp_bary(h);
    r.w0 = h->qw[0];
    if (h->npe != 10) {
        for (int k = 0; k < 4; ++k) r.L[k] = q.L[0][k];
        return r;
    }
    r.a = q.L[1][0];
    r.b = q.L[1][1];
    r.w1 = h->qw[1];
    for (int p = 0; p < 5; ++p) {
        const double* L = q.L[p];
        const double v0 = L[0] * (2 * L[0] - 1), v1 = L[1] * (2 * L[1] - 1);
        const double e01 = 4 * L[0] * L[1], e12 = 4 * L[1] * L[2], e23 = 4 * L[2] * L[3];
        const double w = h->qw[p];
        r.vv += w * v0 * v0;
        r.vw += w * v0 * v1;
        r.ve += w * v0 * e01;
        r.vf += w * v0 * e12;
        r.ee += w * e01 * e01;
        r.ea += w * e01 * e12;
        r.eo += w * e01 * e23;
    }
    return r;
}

}  // namespace tlfea

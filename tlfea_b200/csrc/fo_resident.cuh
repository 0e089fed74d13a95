// fo_resident.cuh -- a Nesterov or AdamW solve in one cooperative launch with every tile of a
// straight-sided mesh resident (SyncedNesterov.cu:97-414, SyncedAdamW.cu:99-425,
// SyncedAdamWNocoop.cu:97-458: the iteration of first_order.cu).
//
// One tile per block.  Nodes are owned by the tiles in even shares (Tiling::own_*).  An inner
// iteration is two phases and two grid barriers:
//
//   tiles   gather the records x and rho (v - v_prev) / dt of the tile's nodes, element forces
//           with the mass term, per-node sums into the node slots;
//   nodes   the owned nodes: force from the slots, gradient, the shares of the norms, and ahead
//           of the stop test (which needs the norms of all blocks) the velocity of the next
//           iteration and its records.  A loop that ends drops them: the velocity it ends with
//           is kept beside.
//
// The node phase's barrier carries the norms, so the stop test costs no barrier of its own.
#pragma once

#include "force_straight.cuh"
#include "grid_barrier.cuh"

namespace tlfea {

struct FOResident {
    double* x4;
    double* w4;
    const int* own_off;
    const int* own_gid;
    const int* node_soff;
    unsigned int* arrived;  // zero at launch
    int* fail;              // set when a bounded wait ran out
    double mass_scale;      // rho / dt
};

// Sums of up to three values over the block, valid in thread 0.
template <int BT>
__device__ __forceinline__ void block_sum3(double (&v)[3], double (*red)[3]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = warp_sum(v[k]);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) red[wid][k] = v[k];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = warp_sum(lane < BT / 32 ? red[lane][k] : 0.0);
    }
}

// Element geometry, loaded where it is used (held across the phases it would cost 20 registers).
template <typename R>
__device__ __forceinline__ void ld_geometry(const R* geo, int tile, R (&ji)[9], R& det) {
    const R* g = geo + (size_t)tile * 10 * TILE_ELEMS + threadIdx.x;
    R v[10];
#pragma unroll
    for (int m = 0; m < 10; ++m) {
        if constexpr (sizeof(R) == 8)
            asm volatile("ld.global.f64 %0, [%1];" : "=d"(v[m]) : "l"(g + m * TILE_ELEMS));
        else
            asm volatile("ld.global.f32 %0, [%1];" : "=f"(v[m]) : "l"(g + m * TILE_ELEMS));
    }
#pragma unroll
    for (int m = 0; m < 9; ++m) ji[m] = v[m];
    det = v[9];
}

// Blocks of BT threads: the element phase uses 128, the node phases all.  FP64 needs 168
// registers (3 blocks of 128 threads per SM, 444 tiles), FP32 128 (4, 592 tiles).  At 15,360
// elements 120 iterations 16 us each against 34 (first_order.cu's persistent kernel: four
// barriers, per-point geometry, nodes gathered per phase).
template <typename R, int NPE, int BT>
__global__ void __launch_bounds__(BT, BT >= 384 ? 1 : (BT >= 192 ? 2 : (sizeof(R) == 4 ? 4 : 3)))
    k_fo_resident(FOArgs S, SeqForceArgs<R> A, FOResident Q) {
    constexpr int TE = TILE_ELEMS;
    constexpr bool DISP = sizeof(R) == 4;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[BT / 32][3];
    __shared__ double sums[3];
    __shared__ int ok_sh;
    const int t = threadIdx.x, tile = blockIdx.x, G = gridDim.x;
    const SForceTables<R>& T = A.T;
    const SForceLayout<R, NPE> L(T.max_local, true);
    R* fe = reinterpret_cast<R*>(smem);
    double* xs = reinterpret_cast<double*>(smem + L.x);
    double* ws = reinterpret_cast<double*>(smem + L.w);
    const unsigned char* tab = smem + L.tab;
    const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
    const uint16_t* lcs = reinterpret_cast<const uint16_t*>(tab + L.lconn);
    const int* slot = reinterpret_cast<const int*>(tab + L.dst);
    const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
    const int* gid = reinterpret_cast<const int*>(tab + L.tab_bytes);  // in the second table buffer
    const uint32_t bar0 = smem_u32(smem + L.bar);
    sf_init_barriers(bar0);
    if (t == 0) {
        sf_issue<R, NPE>(T, L, smem, tile, 0);
        const int pb = T.pad_off[tile];
        const uint32_t bytes = (uint32_t)(T.pad_off[tile + 1] - pb) * sizeof(int);
        mbar_expect_tx(bar0 + 8, bytes);
        bulk_g2s(smem_u32(gid), T.pad_gid + pb, bytes, bar0 + 8);
    }
    bool fine = mbar_wait(bar0, 0);
    fine = __syncthreads_and(mbar_wait(bar0 + 8, 0) && fine);
    if (!fine) {  // (the block leaves below; its copies get one more wait)
        mbar_wait(bar0, 0);
        mbar_wait(bar0 + 8, 0);
    }
    const int nl = T.node_off[tile + 1] - T.node_off[tile];
    const int ob = Q.own_off[tile], no = Q.own_off[tile + 1] - ob;
    const int* own = Q.own_gid + ob;

    unsigned int target = 0;
    // The blocks' shares of n sums (rows k0.. of S.red: other rows than the last meeting's, whose
    // totals some block may still be folding), a barrier, and the totals in `sums`.
    auto meet = [&](double (&v)[3], int n, int k0) -> bool {
        const double* row = S.red + (size_t)k0 * S.red_stride;
        if (n > 0) {
            block_sum3<BT>(v, red);
            if (t == 0)
                for (int k = 0; k < n; ++k) S.red[(size_t)(k0 + k) * S.red_stride + blockIdx.x] = v[k];
        }
        target += (unsigned int)G;
        lin_grid_arrive(Q.arrived);
        if (!lin_grid_wait_sum(Q.arrived, target, row, n > 0 ? G : 0, &ok_sh, &sums[0])) return false;
        if (n > 1) {
            if (t < 32)
                for (int k = 1; k < n; ++k) {
                    double w = 0.0;
                    for (int b = t; b < G; b += 32) w += __ldcg(row + (size_t)k * S.red_stride + b);
                    w = warp_sum(w);
                    if (t == 0) sums[k] = w;
                }
            __syncthreads();
        }
        return true;
    };
    const bool nesterov = S.kind == KIND_NESTEROV, nocoop = S.kind == KIND_ADAMW_NOCOOP;
    const int check = S.check > 0 ? S.check : 1;
    const int eff_outer = (nocoop && S.nc == 0) ? 1 : S.max_outer;

    auto record = [&](int i, const double v[3], const double vp[3], const double xp[3]) {
        double x[3] = {xp[0] + S.dt * v[0], xp[1] + S.dt * v[1], xp[2] + S.dt * v[2]};
        if constexpr (DISP) {
            x[0] -= S.X0x[i];
            x[1] -= S.X0y[i];
            x[2] -= S.X0z[i];
        }
        st_node(Q.x4 + 4 * (size_t)i, x[0], x[1], x[2]);
        st_node(Q.w4 + 4 * (size_t)i, (v[0] - vp[0]) * Q.mass_scale, (v[1] - vp[1]) * Q.mass_scale,
                (v[2] - vp[2]) * Q.mass_scale);
    };
    // AdamW's velocity from (v, g) with the scalars of the iteration (first_order.cu P1)
    struct Scalars {
        double beta, lr, b1t, b2t;
    };
    auto adamw = [&](double v, double g, double m, double va, const Scalars& c, double& mo, double& vo) -> double {
        mo = S.beta1 * m + (1 - S.beta1) * g;
        vo = S.beta2 * va + (1 - S.beta2) * g * g;
        const double mh = nocoop ? mo * c.b1t : mo / c.b1t, vh = nocoop ? vo * c.b2t : vo / c.b2t;
        return v - c.lr * (mh / (sqrt(vh) + S.eps) + S.wd * v);
    };

    for (int o = t; o < no; o += BT) {  // x_prev
        const int i = own[o];
        S.xp[i] = S.x[i];
        S.yp[i] = S.y[i];
        S.zp[i] = S.z[i];
    }
    int outer_flag = 0, status = 0, n_outer = 0, inner_total = 0, last_inner = 0;
    double last_norm = 0.0;
    double* v_end = S.vg;  // the velocity the inner loop ended with
    for (int outer = 0; outer < eff_outer && !outer_flag && !status && fine; ++outer) {
        ++n_outer;
        double tt = 1.0, prev_norm_g = 0.0, norm_g = 0.0, norm_g0 = -1.0, lr = S.lr;
        int inner_flag = 0, inner_count = 0;
        auto scalars = [&](int inner) -> Scalars {  // of inner iteration `inner`, in sequence
            Scalars c{0.0, 0.0, 0.0, 0.0};
            if (nesterov) {
                const double tn = 0.5 * (1.0 + sqrt(1.0 + 4.0 * tt * tt));
                c.beta = (tt - 1.0) / tn;
                tt = tn;
            } else if (nocoop) {
                c.lr = S.lr * pow(S.lr_decay, inner + 1);
                const double tc = (double)(inner + 2);
                c.b1t = 1.0 / (1.0 - pow(S.beta1, tc));
                c.b2t = 1.0 / (1.0 - pow(S.beta2, tc));
            } else {
                lr = lr * S.lr_decay;
                tt += 1;
                c.lr = lr;
                c.b1t = 1 - pow(S.beta1, tt);
                c.b2t = 1 - pow(S.beta2, tt);
            }
            return c;
        };
        // the first iteration's velocity: v itself (Nesterov, beta = 0), AdamW's step from g = 0.
        // AdamW keeps the velocity in two buffers, cur and the next one's.
        double *cur = S.vg, *nxt = S.vk;
        if (S.max_inner > 0) {
            const Scalars c = scalars(0);
            for (int o = t; o < no; o += BT) {
                const int i = own[o];
                const size_t k = 3 * (size_t)i;
                double v[3];
                const double vp[3] = {S.vp[k], S.vp[k + 1], S.vp[k + 2]};
                const double xp[3] = {S.xp[i], S.yp[i], S.zp[i]};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    v[d] = S.vg[k + d];
                    if (nesterov) {
                        S.vk[k + d] = v[d];
                    } else {
                        double mo, vo;
                        v[d] = adamw(v[d], 0.0, 0.0, 0.0, c, mo, vo);
                        S.m[k + d] = mo;
                        S.va[k + d] = vo;
                        S.vg[k + d] = v[d];
                    }
                }
                record(i, v, vp, xp);
            }
        }
        double none[3] = {0.0, 0.0, 0.0};
        if (!(fine = meet(none, 0, 0))) break;
        for (int inner = 0; inner < S.max_inner && !inner_flag; ++inner) {
            ++inner_count;
            // ---- tiles
            R ji[9], det = R(0);
            if (t < TE) ld_geometry(T.geo, tile, ji, det);
            for (int ln = t; ln < nl; ln += BT) {
                double xv[3], wv[3];
                const size_t g = 4 * (size_t)gid[ln];
                ld_node_shared(Q.x4 + g, xv);
                ld_node_shared(Q.w4 + g, wv);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    xs[3 * ln + d] = xv[d];
                    ws[3 * ln + d] = wv[d];
                }
            }
            __syncthreads();
            if (t < TE) {
                int lc[NPE];
#pragma unroll
                for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
                auto xa = [&](int a, int c) { return xs[lc[a] + c]; };
                auto wa = [&](int a, int c) { return ws[lc[a] + c]; };
                svk_element<R, NPE, false, true>(ji, det, A.lambda, A.mu, R(0), R(0), A.rule, xa, wa, wa, fe + t);
            }
            __syncthreads();
            for (int ln = t; ln < nl; ln += BT) {
                double s0, s1, s2;
                tile_node_sum(fe, incs, ln ? iends[ln - 1] : 0, iends[ln], s0, s1, s2);
                st_node(A.slots + 4 * (size_t)slot[ln], s0, s1, s2);
            }
            if (!(fine = meet(none, 0, 0))) break;
            // ---- nodes: gradient, norms, and the next iteration's velocity
            const bool do_check = nesterov || (inner % check == 0);
            const Scalars c = scalars(inner + 1);
            double sm[3] = {0.0, 0.0, 0.0};  // ||g||^2, then ||v_next||^2, ||v_k||^2 or ||v||^2
            for (int o = t; o < no; o += BT) {
                const int i = own[o];
                const size_t k = 3 * (size_t)i;
                const int so = Q.node_soff[i], n = Q.node_soff[i + 1] - so;
                const bool held = S.nc > 0 && S.jt_off[k] != S.jt_off[k + 1];
                double f[3], g[3], v[3], vk[3], mm[3], va[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {  // every load before the first store
                    g[d] = S.f_ext[k + d];
                    v[d] = cur[k + d];
                    vk[d] = nesterov ? S.vk[k + d] : 0.0;
                    mm[d] = nesterov ? 0.0 : S.m[k + d];
                    va[d] = nesterov ? 0.0 : S.va[k + d];
                }
                const double vp[3] = {S.vp[k], S.vp[k + 1], S.vp[k + 2]};
                const double xp[3] = {S.xp[i], S.yp[i], S.zp[i]};
                f[0] = f[1] = f[2] = 0.0;
                for (int j = 0; j < n; j += 4) {  // slots in tile order, four in flight
                    double sv[4][3];
#pragma unroll
                    for (int q = 0; q < 4; ++q) ld_node_shared(A.slots + 4 * (size_t)(so + min(j + q, n - 1)), sv[q]);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (j + q < n) {
#pragma unroll
                            for (int d = 0; d < 3; ++d) f[d] += sv[q][d];
                        }
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) g[d] = f[d] - g[d];
                if (held) {
                    const double xj[3] = {S.xj[i], S.yj[i], S.zj[i]};
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        for (int q = S.jt_off[k + d]; q < S.jt_off[k + d + 1]; ++q)
                            g[d] += S.dt * (S.lam[S.jt_col[q]] + S.rho * (xp[d] + S.dt * v[d] - xj[d]));
                }
                double next[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    sm[0] += g[d] * g[d];
                    if (nesterov) {
                        const double vn = v[d] - S.alpha * g[d];
                        sm[1] += vn * vn;
                        sm[2] += vk[d] * vk[d];
                        S.vk[k + d] = vn;
                        next[d] = vn + c.beta * (vn - vk[d]);
                        S.vg[k + d] = next[d];
                    } else {
                        sm[1] += v[d] * v[d];
                        next[d] = adamw(v[d], g[d], mm[d], va[d], c, mm[d], va[d]);
                        S.m[k + d] = mm[d];
                        S.va[k + d] = va[d];
                        nxt[k + d] = next[d];
                    }
                }
                record(i, next, vp, xp);
            }
            if (!(fine = meet(sm, nesterov ? 3 : 2, 0))) break;
            if (nesterov) {
                norm_g = sqrt(sums[0]);
                if (!isfinite(norm_g)) status = TLFEA_NONFINITE;
                if (inner > 0 && fabs(norm_g - prev_norm_g) < S.inner_tol) inner_flag = 1;
                if (inner > 0 && fabs(sqrt(sums[1]) - sqrt(sums[2])) < S.inner_tol) inner_flag = 1;
                prev_norm_g = norm_g;
                v_end = S.vk;
            } else {
                if (do_check) {
                    norm_g = sqrt(sums[0]);
                    const double nv = sqrt(sums[1]);
                    if (!isfinite(norm_g)) status = TLFEA_NONFINITE;
                    if (norm_g0 < 0.0) norm_g0 = norm_g;
                    const double tol_abs = S.inner_tol * (1.0 + nv);
                    const double tol_rel = (S.rtol > 0.0 && norm_g0 > 0.0) ? (S.rtol * norm_g0) : 0.0;
                    if (norm_g <= tol_abs || (tol_rel > 0.0 && norm_g <= tol_rel)) inner_flag = 1;
                }
                v_end = cur;
                double* w = cur;
                cur = nxt;
                nxt = w;
            }
            if (status) break;
        }
        inner_total += inner_count;
        last_inner = inner_count;
        last_norm = norm_g;
        if (status || !fine) break;
        // ---- outer update: v_prev, constraints, multipliers (the owners of the fixed nodes)
        double sc[3] = {0.0, 0.0, 0.0};
        for (int o = t; o < no; o += BT) {
            const int i = own[o];
            const size_t k = 3 * (size_t)i;
            const double v[3] = {v_end[k], v_end[k + 1], v_end[k + 2]};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                S.vp[k + d] = v[d];
                S.vg[k + d] = v[d];
            }
            if (S.nc > 0 && S.jt_off[k] != S.jt_off[k + 1]) {
                const double xp[3] = {S.xp[i], S.yp[i], S.zp[i]};
                const double xj[3] = {S.xj[i], S.yj[i], S.zj[i]};
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    for (int q = S.jt_off[k + d]; q < S.jt_off[k + d + 1]; ++q) {
                        const int ci = S.jt_col[q];
                        const double cc = xp[d] + S.dt * v[d] - xj[d];
                        S.c[ci] = cc;
                        S.lam[ci] += S.rho * S.dt * cc;
                        sc[0] += cc * cc;
                    }
            }
        }
        v_end = S.vg;
        if (!(fine = meet(sc, 1, 3))) break;
        const double norm_c = sqrt(sums[0]);
        if (nocoop) {
            if (S.nc > 0 && norm_c < S.outer_tol && inner_flag) outer_flag = 1;
        } else if (fabs(norm_c) < S.outer_tol) {
            outer_flag = 1;
        }
    }
    if (!fine) {  // a bounded wait ran out: the positions stay
        if (t == 0) *Q.fail = 1;
        return;
    }
    // final positions x = x_prev + dt v, the force of the last evaluation
    for (int o = t; o < no; o += BT) {
        const int i = own[o];
        const size_t k = 3 * (size_t)i;
        const double v[3] = {v_end[k], v_end[k + 1], v_end[k + 2]};
#pragma unroll
        for (int d = 0; d < 3; ++d) S.vg[k + d] = v[d];
        S.x[i] = S.xp[i] + S.dt * v[0];
        S.y[i] = S.yp[i] + S.dt * v[1];
        S.z[i] = S.zp[i] + S.dt * v[2];
        if (inner_total > 0) {
            double f[3] = {0.0, 0.0, 0.0};
            for (int j = Q.node_soff[i]; j < Q.node_soff[i + 1]; ++j) {
                double sv[3];
                ld_node_shared(A.slots + 4 * (size_t)j, sv);
#pragma unroll
                for (int d = 0; d < 3; ++d) f[d] += sv[d];
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if constexpr (DISP)
                    S.f_int32[k + d] = (float)f[d];
                else
                    S.f_int64[k + d] = f[d];
            }
        }
    }
    if (blockIdx.x == 0 && t == 0) {
        S.stat[0] = n_outer;
        S.stat[1] = inner_total;
        S.stat[2] = last_inner;
        S.stat[3] = status;
        *S.stat_norm = last_norm;
        *S.stat_rel = -1.0;
        S.stat[8] = 0;
    }
}

}  // namespace tlfea

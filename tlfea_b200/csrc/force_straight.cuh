// force_straight.cuh -- tile kernels of the nonlinear force on straight-sided meshes
// (straight_svk.cuh): the single evaluation behind ComputeInternalForce, and the tile loop of
// the first-order solvers and the batched sequences.
//
// Both run resident blocks over the tiles like lin_cg.cuh's product: while one unit is
// computed, the next one's tables arrive by bulk copies, and its geometry and node values are
// in flight in registers.
#pragma once

#include "force_pipe.cuh"
#include "straight_svk.cuh"

namespace tlfea {

// Shared memory: [element forces][node values: 3 or 6 per local node][tables twice][barriers].
template <typename R, int NPE>
struct SForceLayout {
    size_t x, w, tab, inc, lconn, dst, iend, tab_bytes, bar, total;
    __host__ __device__ SForceLayout(int ml, bool six) {
        auto al = [](size_t v) { return (v + 15) & ~size_t(15); };
        x = al(3 * (size_t)NPE * TILE_ELEMS * sizeof(R));
        w = al(x + 3 * (size_t)ml * sizeof(double));
        tab = al(w + (six ? 3 * (size_t)ml * sizeof(double) : 0));
        inc = 0;
        lconn = inc + NPE * TILE_ELEMS * sizeof(uint16_t);
        dst = lconn + NPE * TILE_ELEMS * sizeof(uint16_t);
        iend = dst + (size_t)ml * sizeof(int);
        tab_bytes = al(iend + (size_t)ml * sizeof(uint16_t));
        bar = tab + 2 * tab_bytes;
        total = bar + 16;
    }
};

template <typename R>
struct SForceTables {
    const int* node_off;
    const int* pad_off;
    const int* pad_gid;
    const int* pad_dst;  // scatter destinations, or node slots
    const uint16_t* pad_iend;
    const uint16_t* inc;
    const uint16_t* lconn;
    const R* geo;
    int n_tiles, max_local;
    int* err;
};

template <typename R, int NPE>
__device__ __forceinline__ void sf_issue(const SForceTables<R>& T, const SForceLayout<R, NPE>& L, unsigned char* smem,
                                         int tile, int load) {  // one thread
    constexpr uint32_t TAB = NPE * TILE_ELEMS * sizeof(uint16_t);
    const uint32_t bar = smem_u32(smem + L.bar) + 8 * (load & 1);
    unsigned char* tab = smem + L.tab + (load & 1) * L.tab_bytes;
    const int pb = T.pad_off[tile];
    const uint32_t np = (uint32_t)(T.pad_off[tile + 1] - pb);
    mbar_expect_tx(bar, 2 * TAB + np * (sizeof(int) + sizeof(uint16_t)));
    bulk_g2s(smem_u32(tab + L.inc), T.inc + (size_t)tile * NPE * TILE_ELEMS, TAB, bar);
    bulk_g2s(smem_u32(tab + L.lconn), T.lconn + (size_t)tile * NPE * TILE_ELEMS, TAB, bar);
    bulk_g2s(smem_u32(tab + L.dst), T.pad_dst + pb, np * sizeof(int), bar);
    bulk_g2s(smem_u32(tab + L.iend), T.pad_iend + pb, np * sizeof(uint16_t), bar);
}

template <typename R>
__device__ __forceinline__ void sf_geometry(const SForceTables<R>& T, int tile, R (&ji)[9], R& det) {
    const R* g = T.geo + (size_t)tile * 10 * TILE_ELEMS + threadIdx.x;
#pragma unroll
    for (int m = 0; m < 9; ++m) ji[m] = __ldg(g + m * TILE_ELEMS);
    det = __ldg(g + 9 * TILE_ELEMS);
}

__device__ __forceinline__ void sf_init_barriers(uint32_t bar) {
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
}

// ------------------------------------------------------------------ ComputeInternalForce

template <typename R>
struct SForceArgs {
    SForceTables<R> T;
    const double *x, *y, *z, *X0x, *X0y, *X0z;
    const double* nodes;  // records of x, or of x - X0 (FP32)
    const double* v;  // interleaved velocities (DAMP)
    R* f_out;
    R* partial;
    R lambda, mu, eta, lamd;
    SvkRule rule;
};

// The internal force; REC: node values from records (a 256-bit load a node, FP32: displacements),
// else gathered from the position arrays (FP32: differenced from X0 in FP64), so that nothing has
// to be rebuilt first (the rule stands at the launch); interior nodes written directly, shared
// nodes as per-tile partials for k_combine.  At 480,000 elements, with the positions rewritten
// before each call, a call takes 93 us in FP64 against 161 for the gradient stream and the copy it
// stages from, 78 in FP32 against 118: 15,360 bytes of geometry per tile against 163,840.  What is
// left is shared-memory wavefronts (node values out, forces in, forces summed) and latency.
template <typename R, int NPE, bool DAMP, bool REC>
__global__ void __launch_bounds__(TILE_ELEMS, sizeof(R) == 4 ? (DAMP ? 3 : 4) : (DAMP ? 2 : 3)) k_force_straight(SForceArgs<R> A) {
    constexpr int TE = TILE_ELEMS, NB = NPE == 10 ? 3 : 1;  // node values in flight per thread
    constexpr bool DISP = sizeof(R) == 4 && !REC;
    extern __shared__ __align__(128) unsigned char smem[];
    const int t = threadIdx.x;
    const SForceTables<R>& T = A.T;
    const SForceLayout<R, NPE> L(T.max_local, DAMP);
    R* fe = reinterpret_cast<R*>(smem);
    double* xs = reinterpret_cast<double*>(smem + L.x);
    double* vs = reinterpret_cast<double*>(smem + L.w);
    const uint32_t bar0 = smem_u32(smem + L.bar);
    sf_init_barriers(bar0);
    int tile = blockIdx.x;
    if (t == 0) sf_issue<R, NPE>(T, L, smem, tile, 0);
    R ji[9], det;
    double pv[NB][3], p0[DISP ? NB : 1][3];
    int nl = T.node_off[tile + 1] - T.node_off[tile];
    auto gather = [&](int tl, int n) {
        const int pb = T.pad_off[tl];
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int g = T.pad_gid[pb + min(t + j * TE, n - 1)];
            if constexpr (REC) {
                ld_node(A.nodes + 4 * (size_t)g, pv[j]);
            } else {
                pv[j][0] = A.x[g];
                pv[j][1] = A.y[g];
                pv[j][2] = A.z[g];
            }
            if constexpr (DISP) {
                p0[j][0] = A.X0x[g];
                p0[j][1] = A.X0y[g];
                p0[j][2] = A.X0z[g];
            }
        }
    };
    sf_geometry(T, tile, ji, det);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    gather(tile, nl);
    for (int it = 0; tile < T.n_tiles; ++it) {
        const bool landed = mbar_wait(bar0 + 8 * (it & 1), (it >> 1) & 1);
        const unsigned char* tab = smem + L.tab + (it & 1) * L.tab_bytes;
        const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
        const uint16_t* lcs = reinterpret_cast<const uint16_t*>(tab + L.lconn);
        const int* dst = reinterpret_cast<const int*>(tab + L.dst);
        const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int ln = t + j * TE;
            if (ln < nl) {
#pragma unroll
                for (int d = 0; d < 3; ++d) xs[3 * ln + d] = DISP ? pv[j][d] - p0[DISP ? j : 0][d] : pv[j][d];
            }
        }
        if (DAMP || nl > NB * TE) {
            const int pb = T.pad_off[tile];
            for (int ln = t; ln < nl; ln += TE) {
                const int g = T.pad_gid[pb + ln];
                if (REC && ln >= NB * TE) {  // larger tiles
                    double p[3];
                    ld_node(A.nodes + 4 * (size_t)g, p);
#pragma unroll
                    for (int d = 0; d < 3; ++d) xs[3 * ln + d] = p[d];
                } else if (ln >= NB * TE) {
                    xs[3 * ln + 0] = A.x[g] - (DISP ? A.X0x[g] : 0.0);
                    xs[3 * ln + 1] = A.y[g] - (DISP ? A.X0y[g] : 0.0);
                    xs[3 * ln + 2] = A.z[g] - (DISP ? A.X0z[g] : 0.0);
                }
                if constexpr (DAMP) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) vs[3 * ln + d] = A.v[3 * (size_t)g + d];
                }
            }
        }
        // values staged; the other table buffer's readers are past it
        if (!__syncthreads_and(landed)) {
            tables_late(T.err, bar0 + 8 * (it & 1), (it >> 1) & 1);
            return;
        }
        const int next = tile + gridDim.x;
        if (t == 0 && next < T.n_tiles) sf_issue<R, NPE>(T, L, smem, next, it + 1);
        {
            int lc[NPE];
#pragma unroll
            for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
            auto xa = [&](int a, int c) { return xs[lc[a] + c]; };
            auto va = [&](int a, int c) { return vs[lc[a] + c]; };
            svk_element<R, NPE, DAMP, false>(ji, det, A.lambda, A.mu, A.eta, A.lamd, A.rule, xa, va, va, fe + t);
        }
        const int nl_now = nl;
        if (next < T.n_tiles) {  // in flight during the scatter
            nl = T.node_off[next + 1] - T.node_off[next];
            sf_geometry(T, next, ji, det);
            gather(next, nl);
        }
        __syncthreads();  // element forces complete
        for (int ln = t; ln < nl_now; ln += TE) {
            double s0, s1, s2;
            tile_node_sum(fe, incs, ln ? iends[ln - 1] : 0, iends[ln], s0, s1, s2);
            const int dn = dst[ln];
            R* o = dn >= 0 ? A.f_out + 3 * (size_t)dn : A.partial + 3 * (size_t)(-dn - 1);
            o[0] = R(s0);
            o[1] = R(s1);
            o[2] = R(s2);
        }
        // every thread's reads of the tables precede the bulk copies that replace them
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();  // forces, values and tables free
        tile = next;
    }
    // outputs written: the combine kernel (a programmatic dependent) may be scheduled
    asm volatile("griddepcontrol.launch_dependents;");
}

// ------------------------------------------------------------------ solvers

// Node values of one or many sequences as records: x (FP64: positions; FP32: displacements) and
// w = rho (v - v_prev) / dt, sequence s at node_stride * s nodes; tile sums into node slots.
template <typename R>
struct SeqForceArgs {
    SForceTables<R> T;  // pad_dst = node slots
    const double* x;
    const double* w;
    double* slots;
    int n_seq, group;  // sequences per pass of a tile's tables
    long long node_stride, slot_stride;
    const double* lam_s;  // per sequence, or null: lambda, mu
    const double* mu_s;
    R lambda, mu;
    SvkRule rule;
};

// Forces and the mass term over the tiles and the running sequences.  A block's work is a
// sequence of units (item, sequence), an item a tile and a group of sequences.  False (in every
// thread) if a table did not land.
template <typename R, int NPE, typename Run>
__device__ __forceinline__ bool seq_force_tiles(const SeqForceArgs<R>& A, unsigned char* smem, Run running) {
    constexpr int TE = TILE_ELEMS, NB = NPE == 10 ? 3 : 1;  // node values in flight per thread
    const int t = threadIdx.x;
    const SForceTables<R>& T = A.T;
    const SForceLayout<R, NPE> L(T.max_local, true);
    R* fe = reinterpret_cast<R*>(smem);
    double* xs = reinterpret_cast<double*>(smem + L.x);
    double* ws = reinterpret_cast<double*>(smem + L.w);
    const uint32_t bar0 = smem_u32(smem + L.bar);
    const int groups = (A.n_seq + A.group - 1) / A.group;
    const int n_items = T.n_tiles * groups;  // tile-major: the sequences of a tile run back to back
    auto seek = [&](int& item, int& seq) {
        for (; item < n_items; item += gridDim.x) {
            const int g0 = (item % groups) * A.group, g1 = min(g0 + A.group, A.n_seq);
            for (seq = max(seq, g0); seq < g1; ++seq)
                if (running(seq)) return;
            seq = 0;
        }
        item = n_items;
    };
    R ji[9], det;
    double xv[NB][3], wv[NB][3];
    auto gather = [&](int tile, int seq, int n) {
        const int pb = T.pad_off[tile];
        const size_t o = 4 * (size_t)seq * A.node_stride;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const size_t g = o + 4 * (size_t)T.pad_gid[pb + min(t + j * TE, n - 1)];
            ld_node(A.x + g, xv[j]);
            ld_node(A.w + g, wv[j]);
        }
    };
    int item = blockIdx.x, seq = 0, load = 0;
    seek(item, seq);
    if (item >= n_items) return true;
    int tile = item / groups;
    int nl = T.node_off[tile + 1] - T.node_off[tile];
    if (t == 0) sf_issue<R, NPE>(T, L, smem, tile, 0);
    sf_geometry(T, tile, ji, det);
    gather(tile, seq, nl);
    bool fresh = true;
    while (item < n_items) {
        const bool landed = !fresh || mbar_wait(bar0 + 8 * (load & 1), (load >> 1) & 1);
        const unsigned char* tab = smem + L.tab + (load & 1) * L.tab_bytes;
        const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
        const uint16_t* lcs = reinterpret_cast<const uint16_t*>(tab + L.lconn);
        const int* slot = reinterpret_cast<const int*>(tab + L.dst);
        const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int ln = t + j * TE;
            if (ln < nl) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    xs[3 * ln + d] = xv[j][d];
                    ws[3 * ln + d] = wv[j][d];
                }
            }
        }
        for (int ln = t + NB * TE; ln < nl; ln += TE) {  // larger tiles
            const size_t g = 4 * ((size_t)seq * A.node_stride + T.pad_gid[T.pad_off[tile] + ln]);
            ld_node(A.x + g, xv[0]);
            ld_node(A.w + g, wv[0]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                xs[3 * ln + d] = xv[0][d];
                ws[3 * ln + d] = wv[0][d];
            }
        }
        int item2 = item, seq2 = seq + 1;
        seek(item2, seq2);
        const bool more = item2 < n_items, swap = more && item2 != item;
        const int tile2 = more ? item2 / groups : tile;
        const R lam = A.lam_s ? R(__ldg(A.lam_s + seq)) : A.lambda, mu = A.lam_s ? R(__ldg(A.mu_s + seq)) : A.mu;
        // values staged; the other table buffer's readers are past it
        if (!__syncthreads_and(landed)) {
            tables_late(T.err, bar0 + 8 * (load & 1), (load >> 1) & 1);
            return false;
        }
        if (swap && t == 0) sf_issue<R, NPE>(T, L, smem, tile2, load + 1);
        {
            int lc[NPE];
#pragma unroll
            for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
            auto xa = [&](int a, int c) { return xs[lc[a] + c]; };
            auto wa = [&](int a, int c) { return ws[lc[a] + c]; };
            svk_element<R, NPE, false, true>(ji, det, lam, mu, R(0), R(0), A.rule, xa, wa, wa, fe + t);
        }
        const int nl_now = nl;
        if (more) {  // in flight during the scatter
            if (swap) {
                nl = T.node_off[tile2 + 1] - T.node_off[tile2];
                sf_geometry(T, tile2, ji, det);
            }
            gather(tile2, seq2, nl);
        }
        __syncthreads();  // element forces complete
        double* slots = A.slots + 4 * (size_t)seq * A.slot_stride;
        for (int ln = t; ln < nl_now; ln += TE) {
            double s0, s1, s2;
            tile_node_sum(fe, incs, ln ? iends[ln - 1] : 0, iends[ln], s0, s1, s2);
            st_node(slots + 4 * (size_t)slot[ln], s0, s1, s2);
        }
        // every thread's reads of the tables precede the bulk copies that replace them
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();  // forces, values and tables free
        fresh = swap;
        if (swap) ++load;
        item = item2;
        seq = seq2;
        tile = tile2;
    }
    return true;
}

// A node's slots [b, e) summed in tile order, two in flight.
__device__ __forceinline__ void node_slot_sum(const double* slots, int b, int e, double f[3]) {
    f[0] = f[1] = f[2] = 0.0;
    for (int k = b; k < e; k += 2) {
        double v[2][3];
        ld_node(slots + 4 * (size_t)k, v[0]);
        ld_node(slots + 4 * (size_t)min(k + 1, e - 1), v[1]);
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d] += v[0][d];
        if (k + 1 < e) {
#pragma unroll
            for (int d = 0; d < 3; ++d) f[d] += v[1][d];
        }
    }
}

template <typename R>
inline SForceTables<R> sforce_tables(const tlfea_element_s* h, bool slots) {
    const Tiling& tl = h->tl;
    SForceTables<R> T{};
    T.node_off = tl.node_off;
    T.pad_off = tl.pad_off;
    T.pad_gid = tl.pad_gid;
    T.pad_dst = slots ? tl.pad_slot : tl.pad_dst;
    T.pad_iend = tl.pad_iend;
    T.inc = tl.inc;
    T.lconn = tl.lconn;
    if constexpr (sizeof(R) == 8)
        T.geo = tl.geo64;
    else
        T.geo = tl.geo32;
    T.n_tiles = tl.n_tiles;
    T.max_local = tl.max_local_pad;
    T.err = h->d_err;
    return T;
}

}  // namespace tlfea

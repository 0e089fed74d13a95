// lin_cg.cuh -- LinearStaticSolver's CG at the reference configuration on straight-sided
// elements (new: the reference assembles K, LinearStaticSolver.cu:196-263).
//
// A first solve starts from the undeformed mesh: F = I, S = 0, and K is the linear
// elasticity operator.  With one Jacobian per element (straight.cuh) its product needs 80
// bytes of geometry per element, so K is neither assembled nor streamed:
//
//   element tiles   p gathered from node order, ten nodal forces per element, per-node sums
//                   in the tile's incidence order into the node's slots (no atomics); the
//                   tile's share of p.Kp is sum_nodes p . (tile sum): alpha needs no
//                   completed q;
//   node update     q = the node's slots in tile order; r -= alpha q, r.r, the stop test and
//                   beta;
//   direction       u += alpha p, p = r + beta p.
//
// Two forms of the same arithmetic.  k_lin_cg: one cooperative launch for the whole solve,
// one tile per block, every tile resident (4 blocks per SM: up to 592 tiles, 75,776
// elements): geometry in registers, p of the tile's nodes in shared memory, the direction
// folded into the next gather, so an iteration is two grid barriers.  Its blocks have 512
// threads while there is a tile per SM or fewer, 256 up to two, else 128: the element phase
// uses 128, the node phases all.  k_lin_tiles /
// k_lin_update / k_lin_direction: one launch per phase in CUDA-graph chunks for larger
// meshes.
//
// Fixed DOFs: f, and so r and p, are zero there throughout; their rows are skipped.
#pragma once

#include "force_pipe.cuh"
#include "grid_barrier.cuh"
#include "solver.cuh"
#include "straight.cuh"

namespace tlfea {

struct LinArgs {
    int N, n_tiles, max_local;  // max_local: the node record's padded tile size
    const int* node_off;
    const int* pad_off;
    const int* pad_gid;
    const int* pad_slot;
    const uint16_t* pad_iend;
    const uint16_t* inc;
    const uint16_t* lconn;
    const double* geo;
    const int* node_soff;
    const int* own_off;
    const int* own_gid;
    const uint16_t* own_ln;
    const unsigned char* is_fixed;  // 3N
    const double* f;
    double* u;
    double* r;      // 3N; the resident solve: 4 per node (ld_node)
    double* p;      // 4 per node (ld_node)
    double* slots;  // 4 per node slot
    double* part;   // partial sums: blocks of the tiles, of the update (resident: 2 * n_tiles)
    double lambda, mu, tol;
    int max_iter;
    LinRule rule;
    CgCtl* ctl;
};

// Shared memory of a tile: [element forces][p][tables: incidence, local connectivity, slots,
// incidence ends, node ids; twice in the pipelined tile kernel][barriers].
template <int NPE>
struct LinLayout {
    size_t p, tab, inc, lconn, slot, iend, gid, tab_bytes, bar, total;
    __host__ __device__ LinLayout(int ml, int buffers) {
        auto al = [](size_t v) { return (v + 15) & ~size_t(15); };
        p = 3 * (size_t)NPE * TILE_ELEMS * sizeof(double);
        tab = al(p + 3 * (size_t)ml * sizeof(double));
        inc = 0;
        lconn = inc + NPE * TILE_ELEMS * sizeof(uint16_t);
        slot = lconn + NPE * TILE_ELEMS * sizeof(uint16_t);
        iend = slot + (size_t)ml * sizeof(int);
        gid = al(iend + (size_t)ml * sizeof(uint16_t));
        tab_bytes = buffers == 1 ? gid + (size_t)ml * sizeof(int) : gid;  // the pipeline reads node ids ahead
        bar = tab + buffers * tab_bytes;
        total = bar + 16;
    }
};

__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// bulk_g2s of data that is to leave L2 first.
__device__ __forceinline__ void bulk_g2s_stream(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar,
                                                uint64_t pol) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            dst),
        "l"(src), "r"(bytes), "r"(bar), "l"(pol)
        : "memory");
}

// The tables of a tile into `tab` by bulk copies onto `bar` (one thread; `bar` initialised
// with count 1).
template <int NPE, bool STREAM>
__device__ __forceinline__ void lin_issue_tables(const LinArgs& A, int tile, unsigned char* tab,
                                                 const LinLayout<NPE>& L, uint32_t bar) {
    constexpr uint32_t TAB = NPE * TILE_ELEMS * sizeof(uint16_t);
    const int pb = A.pad_off[tile];
    const uint32_t np = (uint32_t)(A.pad_off[tile + 1] - pb);
    mbar_expect_tx(bar, 2 * TAB + np * (sizeof(int) + sizeof(uint16_t) + (STREAM ? 0 : sizeof(int))));
    auto copy = [&](size_t to, const void* src, uint32_t bytes) {
        if constexpr (STREAM)
            bulk_g2s_stream(smem_u32(tab + to), src, bytes, bar, evict_first_policy());
        else
            bulk_g2s(smem_u32(tab + to), src, bytes, bar);
    };
    copy(L.inc, A.inc + (size_t)tile * NPE * TILE_ELEMS, TAB);
    copy(L.lconn, A.lconn + (size_t)tile * NPE * TILE_ELEMS, TAB);
    copy(L.slot, A.pad_slot + pb, np * sizeof(int));
    copy(L.iend, A.pad_iend + pb, np * sizeof(uint16_t));
    if constexpr (!STREAM) copy(L.gid, A.pad_gid + pb, np * sizeof(int));  // the pipeline reads node ids ahead
}

// J^-1 and det J of the element in lane t of a tile.  STREAM (the launches per phase, at every
// size they run at): the tables and the geometry are read once per iteration and marked to leave
// L2 first, so that the vectors stay.  An iteration marked / unmarked: 109.8 / 113.1 us at 3,750
// tiles, 70.3 / 72.7 at 2,279, and where everything fits 46.3 / 45.5 at 1,200, 36.6 / 36.0 at 610.
template <bool STREAM>
__device__ __forceinline__ void ld_geo(const double* geo, int tile, int t, double ji[9], double& det) {
    const double* g = geo + (size_t)tile * 10 * TILE_ELEMS + t;
    double v[10];
    if constexpr (STREAM) {
        const uint64_t pol = evict_first_policy();
#pragma unroll
        for (int m = 0; m < 10; ++m)
            asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;"
                         : "=d"(v[m])
                         : "l"(g + m * TILE_ELEMS), "l"(pol));
    } else {
#pragma unroll
        for (int m = 0; m < 10; ++m) asm volatile("ld.global.f64 %0, [%1];" : "=d"(v[m]) : "l"(g + m * TILE_ELEMS));
    }
#pragma unroll
    for (int m = 0; m < 9; ++m) ji[m] = v[m];
    det = v[9];
}

// The tile's element forces (in fe) summed per local node into the node's slot; returns
// this thread's share of p . K p.
__device__ __forceinline__ double lin_scatter(const double* fe, const double* ps, const uint16_t* incs,
                                              const uint16_t* iends, const int* slot, int nl, double* slots) {
    double dot = 0.0;
    for (int ln = threadIdx.x; ln < nl; ln += blockDim.x) {
        const int beg = ln ? iends[ln - 1] : 0;
        const int end = iends[ln];
        double s0, s1, s2;
        tile_node_sum(fe, incs, beg, end, s0, s1, s2);
        st_node(slots + 4 * (size_t)slot[ln], s0, s1, s2);
        dot += ps[3 * ln + 0] * s0 + ps[3 * ln + 1] * s1 + ps[3 * ln + 2] * s2;
    }
    return dot;
}

// ctl->deformed = 1 unless the positions are the reference configuration, bit for bit.
__global__ void k_at_reference(int N, const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, const double* __restrict__ X0x,
                               const double* __restrict__ X0y, const double* __restrict__ X0z, CgCtl* ctl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool moved = i < N && !(x[i] == X0x[i] && y[i] == X0y[i] && z[i] == X0z[i]);
    if (__syncthreads_or(moved) && threadIdx.x == 0) ctl->deformed = 1;
}

// Sum over the block, in every thread (warps in order); `red` holds a value per warp.
__device__ __forceinline__ double block_sum_all(double v, double* red) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    return s;
}

// A node's slots [b, b + n) summed in slot (tile) order, four in flight (most shared nodes
// have two to four).
__device__ __forceinline__ void lin_slot_sum(const double* slots, int b, int n, double q[3]) {
    q[0] = q[1] = q[2] = 0.0;
    for (int k = 0; k < n; k += 4) {
        double v[4][3];
#pragma unroll
        for (int i = 0; i < 4; ++i) ld_node_shared(slots + 4 * (size_t)(b + min(k + i, n - 1)), v[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (k + i < n) {
#pragma unroll
                for (int d = 0; d < 3; ++d) q[d] += v[i][d];
            }
    }
}

// The whole solve, one tile per resident block (cooperative launch of n_tiles blocks of BT
// threads).  Per iteration: gather p = r + beta p, element forces, slots, barrier, alpha
// (every warp folds the tiles' shares in the same order), update of the owned nodes,
// barrier, the stop test and beta.  Bound by that chain of latencies (at 40x8x8, 120 tiles, in
// cycles: gather 1,800, elements 2,500, scatter 2,100, update 2,500, the two barriers with
// their sums 5,000 each): 10.6 us an iteration, against 27 us of the assembled K's three
// launches.  What mattered: loads issued together before the first store (27,000 cycles for
// the update alone otherwise, the stores ordering the loads), 32-byte node records, owned
// nodes spread evenly over the tiles, one warp folding the sums.
template <int NPE, int BT>
__global__ void __launch_bounds__(BT, 512 / BT) k_lin_cg(LinArgs A) {
    constexpr int TE = TILE_ELEMS;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[32];
    __shared__ double sum_sh;
    __shared__ int ok_sh;
    CgCtl* ctl = A.ctl;
    if (__ldcg(&ctl->deformed)) return;  // uniform over the grid: set before this launch
    const int tile = blockIdx.x, t = threadIdx.x, G = gridDim.x;
    const LinLayout<NPE> L(A.max_local, 1);
    double* fe = reinterpret_cast<double*>(smem);
    double* ps = reinterpret_cast<double*>(smem + L.p);
    unsigned char* tab = smem + L.tab;
    const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
    const uint16_t* lcs = reinterpret_cast<const uint16_t*>(tab + L.lconn);
    const int* slot = reinterpret_cast<const int*>(tab + L.slot);
    const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
    const int* gid = reinterpret_cast<const int*>(tab + L.gid);
    const uint32_t bar = smem_u32(smem + L.bar);
    if (t == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lin_issue_tables<NPE, false>(A, tile, tab, L, bar);
    }
    const int nl = A.node_off[tile + 1] - A.node_off[tile];
    const int ob = A.own_off[tile], no = A.own_off[tile + 1] - ob;
    const int* own_gid = A.own_gid + ob;
    const uint16_t* own_ln = A.own_ln + ob;
    __syncthreads();  // barrier initialised
    bool fine = __syncthreads_and(mbar_wait(bar, 0));
    if (!fine) mbar_wait(bar, 0);  // (the block leaves below; its copies get one more wait)
    for (int k = t; k < 3 * nl; k += BT) ps[k] = 0.0;
    // owned nodes: r = f, u = 0
    double s = 0.0;
    for (int o = t; o < no; o += BT) {
        const int g = own_gid[o];
        const double* fg = A.f + 3 * (size_t)g;  // zero at fixed DOFs
        const double fi[3] = {fg[0], fg[1], fg[2]};
        st_node(A.r + 4 * (size_t)g, fi[0], fi[1], fi[2]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            A.u[3 * (size_t)g + d] = 0.0;
            s += fi[d] * fi[d];
        }
    }
    double* part_a = A.part;
    double* part_b = A.part + G;
    unsigned int target = 0;
    auto post = [&](double v, double* part) {  // the block's share, then its arrival
        const double bs = block_sum(v, red);
        if (t == 0) part[blockIdx.x] = bs;
        target += (unsigned int)G;
        lin_grid_arrive(&ctl->arrived);
    };
    auto wait_sum = [&](const double* part) {
        return lin_grid_wait_sum(&ctl->arrived, target, part, G, &ok_sh, &sum_sh);
    };
    post(s, part_b);
    fine = wait_sum(part_b) && fine;
    const double rr0 = sum_sh;
    double rr = rr0, beta = 0.0, rel = 1.0;
    int iters = 0, status = 0;
    if (rr0 == 0.0)
        rel = 0.0;
    else if (A.max_iter <= 0)
        status = 2;
    else {
        constexpr int NB = BT == 128 ? 3 : (BT == 256 ? 2 : 1);  // gathers in flight per thread
        while (fine) {
            double ji[9], det = 0.0;
            if (t < TE) ld_geo<false>(A.geo, tile, t, ji, det);  // with the gather in flight, not held across the phases
            for (int l0 = t; l0 < nl; l0 += NB * BT) {
                double rv[NB][3];
#pragma unroll
                for (int j = 0; j < NB; ++j) ld_node_shared(A.r + 4 * (size_t)gid[min(l0 + j * BT, nl - 1)], rv[j]);
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    const int ln = l0 + j * BT;
                    if (ln < nl) {
#pragma unroll
                        for (int d = 0; d < 3; ++d) ps[3 * ln + d] = rv[j][d] + beta * ps[3 * ln + d];
                    }
                }
            }
            __syncthreads();
            if (t < TE) {
                int lc[NPE];
#pragma unroll
                for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
                lin_element<double, NPE>(ji, det, A.lambda, A.mu, A.rule, [&](int a, int c) { return ps[lc[a] + c]; },
                                         fe + t);
            }
            __syncthreads();
            post(lin_scatter(fe, ps, incs, iends, slot, nl, A.slots), part_a);
            if (!(fine = wait_sum(part_a))) break;
            const double pq = sum_sh;
            if (pq <= 0.0) {
                status = 1;
                break;
            }
            const double alpha = rr / pq;
            s = 0.0;
            for (int o = t; o < no; o += BT) {
                const int g = own_gid[o];
                const bool fx = A.is_fixed[3 * (size_t)g] != 0;
                const int so = A.node_soff[g], n = A.node_soff[g + 1] - so;
                double rv[3], q[3];
                ld_node_shared(A.r + 4 * (size_t)g, rv);
                lin_slot_sum(A.slots, so, n, q);
                if (fx) continue;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    rv[d] -= alpha * q[d];
                    s += rv[d] * rv[d];
                }
                st_node(A.r + 4 * (size_t)g, rv[0], rv[1], rv[2]);
            }
            post(s, part_b);
            // u += alpha p while the other blocks arrive (p is this block's own copy; zero at
            // fixed DOFs)
            for (int o = t; o < no; o += BT) {
                double* ug = A.u + 3 * (size_t)own_gid[o];
                const double* pl = ps + 3 * own_ln[o];
                const double uv[3] = {ug[0], ug[1], ug[2]};
#pragma unroll
                for (int d = 0; d < 3; ++d) ug[d] = uv[d] + alpha * pl[d];
            }
            if (!(fine = wait_sum(part_b))) break;
            const double rrn = sum_sh;
            rel = sqrt(rrn / rr0);
            ++iters;
            if (rel < A.tol) break;
            beta = rrn / rr;
            rr = rrn;
            if (iters >= A.max_iter) {
                status = 2;
                break;
            }
        }
    }
    if (t == 0 && !fine) ctl->status = 3;  // a bounded wait ran out
    if (blockIdx.x == 0 && t == 0 && fine) {
        ctl->rr0 = rr0;
        ctl->rel = rel;
        ctl->iters = iters;
        ctl->status = status;
        ctl->done = 1;
    }
}

// ---- one launch per phase.  Each kernel waits for its predecessor (programmatic dependent
// launch) after what does not depend on it: tables, geometry, node ids.

// Last block to arrive (ticket): folds `n` partials in order; the total in thread 0.
__device__ __forceinline__ bool lin_last_fold(double v, double* part, int n, unsigned int* ticket, double* red,
                                              bool* last_sh, double* out) {
    const double bs = block_sum_all(v, red);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = bs;
        __threadfence();
        *last_sh = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!*last_sh) return false;
    __threadfence();
    double w = 0.0;
    for (int b = threadIdx.x; b < n; b += blockDim.x) w += __ldcg(part + b);
    *out = block_sum_all(w, red);
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// K p of the tiles into the node slots; the last block sets alpha.  Resident blocks loop over
// the tiles: while one is computed, the next one's tables arrive by bulk copies, its geometry
// and p are in flight in registers, so a tile costs its arithmetic and its shared-memory
// passes, not its latencies.
template <int NPE>
__global__ void __launch_bounds__(TILE_ELEMS, 4) k_lin_tiles(LinArgs A, int* err) {
    constexpr int TE = TILE_ELEMS, NB = 3;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[4];
    __shared__ bool last_sh;
    asm volatile("griddepcontrol.launch_dependents;");
    CgCtl* ctl = A.ctl;
    const int t = threadIdx.x;
    const LinLayout<NPE> L(A.max_local, 2);
    double* fe = reinterpret_cast<double*>(smem);
    double* ps = reinterpret_cast<double*>(smem + L.p);
    const uint32_t bar0 = smem_u32(smem + L.bar);
    if (t == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lin_issue_tables<NPE, true>(A, blockIdx.x, smem + L.tab, L, bar0);
    }
    double ji[9], det, pv[NB][3];
    int nl = A.node_off[blockIdx.x + 1] - A.node_off[blockIdx.x];
    ld_geo<true>(A.geo, blockIdx.x, t, ji, det);
    // p of this thread's first NB local nodes of a tile
    auto gather = [&](int tile, int n) {
        const int pb = A.pad_off[tile];
        int g[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) g[j] = A.pad_gid[pb + min(t + j * TE, n - 1)];
#pragma unroll
        for (int j = 0; j < NB; ++j) ld_node(A.p + 4 * (size_t)g[j], pv[j]);
    };
    __syncthreads();  // barriers initialised
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool done = __ldcg(&ctl->done) != 0;  // uniform: written by a previous kernel
    double dot = 0.0;
    if (!done) gather(blockIdx.x, nl);
    int it = 0;
    for (int tile = blockIdx.x; tile < A.n_tiles; tile += gridDim.x, ++it) {
        const unsigned char* tab = smem + L.tab + (it & 1) * L.tab_bytes;
        const bool landed = mbar_wait(bar0 + 8 * (it & 1), (it >> 1) & 1);
        if (done) return;  // (the copy in flight has landed)
        const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
        const uint16_t* lcs = reinterpret_cast<const uint16_t*>(tab + L.lconn);
        const int* slot = reinterpret_cast<const int*>(tab + L.slot);
        const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int ln = t + j * TE;
            if (ln < nl) {
#pragma unroll
                for (int d = 0; d < 3; ++d) ps[3 * ln + d] = pv[j][d];
            }
        }
        for (int ln = t + NB * TE; ln < nl; ln += TE) {  // larger tiles
            ld_node(A.p + 4 * (size_t)A.pad_gid[A.pad_off[tile] + ln], pv[0]);
#pragma unroll
            for (int d = 0; d < 3; ++d) ps[3 * ln + d] = pv[0][d];
        }
        // p staged; the other table buffer's readers are past it
        if (!__syncthreads_and(landed)) {
            if (t == 0) {
                ctl->status = 3;
                ctl->done = 1;  // ends the solve: this launch sets no alpha
            }
            tables_late(err, bar0 + 8 * (it & 1), (it >> 1) & 1);
            return;
        }
        const int next = tile + gridDim.x;
        if (t == 0 && next < A.n_tiles) {
            lin_issue_tables<NPE, true>(A, next, smem + L.tab + ((it + 1) & 1) * L.tab_bytes, L,
                                        bar0 + 8 * ((it + 1) & 1));
        }
        {
            int lc[NPE];
#pragma unroll
            for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
            lin_element<double, NPE>(ji, det, A.lambda, A.mu, A.rule, [&](int a, int c) { return ps[lc[a] + c]; },
                                     fe + t);
        }
        const int nl_now = nl;
        if (next < A.n_tiles) {  // in flight during the scatter
            nl = A.node_off[next + 1] - A.node_off[next];
            ld_geo<true>(A.geo, next, t, ji, det);
            gather(next, nl);
        }
        __syncthreads();  // element forces complete
        dot += lin_scatter(fe, ps, incs, iends, slot, nl_now, A.slots);
        // every thread's reads of the tables precede the bulk copies that replace them
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();  // fe, ps and the tables free
    }
    double pq;
    if (lin_last_fold(dot, A.part, (int)gridDim.x, &ctl->ticket, red, &last_sh, &pq) && t == 0) {
        ctl->pq = pq;
        if (pq <= 0.0) {
            ctl->status = 1;
            ctl->done = 1;
        } else {
            ctl->alpha = ctl->rr / pq;
        }
    }
}

// Node i's q = K p from its slots (tile order), two in flight.
__device__ __forceinline__ void lin_node_sum(const double* slots, int b, int e, double q[3]) {
    q[0] = q[1] = q[2] = 0.0;
    for (int k = b; k < e; k += 2) {
        double v[2][3];
        ld_node(slots + 4 * (size_t)k, v[0]);
        ld_node(slots + 4 * (size_t)min(k + 1, e - 1), v[1]);
#pragma unroll
        for (int d = 0; d < 3; ++d) q[d] += v[0][d];
        if (k + 1 < e) {
#pragma unroll
            for (int d = 0; d < 3; ++d) q[d] += v[1][d];
        }
    }
}

// r -= alpha q, r.r; the last block applies the stop test and sets beta
// (LinearStaticSolver.cu:534-557).  Resident blocks, two nodes per thread at a time: a block
// that ends pays the reduction's fence and ticket (about 2 us), so few blocks end.
constexpr int LIN_NODE_THREADS = 256;
__global__ void __launch_bounds__(LIN_NODE_THREADS) k_lin_update(LinArgs A) {
    __shared__ double red[LIN_NODE_THREADS / 32];
    __shared__ bool last_sh;
    asm volatile("griddepcontrol.launch_dependents;");
    CgCtl* ctl = A.ctl;
    const int stride = gridDim.x * blockDim.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (__ldcg(&ctl->done)) return;
    const double alpha = __ldcg(&ctl->alpha);
    double s = 0.0;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < A.N; i0 += 2 * stride) {
        int so[2], se[2];
        bool ok[2];
        double rv[2][3], q[2][3];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = min(i0 + j * stride, A.N - 1);
            so[j] = A.node_soff[i];
            se[j] = A.node_soff[i + 1];
            ok[j] = i0 + j * stride < A.N && !A.is_fixed[3 * (size_t)i];
#pragma unroll
            for (int d = 0; d < 3; ++d) rv[j][d] = A.r[3 * (size_t)i + d];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) lin_node_sum(A.slots, so[j], se[j], q[j]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (!ok[j]) continue;
            const size_t k = 3 * (size_t)(i0 + j * stride);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double ri = rv[j][d] - alpha * q[j][d];
                A.r[k + d] = ri;
                s += ri * ri;
            }
        }
    }
    double rrn;
    if (lin_last_fold(s, A.part, (int)gridDim.x, &ctl->ticket, red, &last_sh, &rrn) && threadIdx.x == 0) {
        const double rel = (ctl->rr0 > 0.0) ? sqrt(rrn / ctl->rr0) : sqrt(rrn);
        ctl->iters += 1;
        if (rel < A.tol) {
            ctl->rel = rel;
            ctl->done = 2;  // k_lin_direction still owes this iteration's u
        } else {
            ctl->beta = rrn / ctl->rr;
            ctl->rr = rrn;
            if (ctl->iters >= A.max_iter) {
                ctl->rel = rel;
                ctl->status = 2;
                ctl->done = 2;
            }
        }
    }
}

// u += alpha p, then p = r + beta p: the one kernel that reads p by nodes.  An iteration that
// ended the solve (done = 2) still gets its u; the last block then closes it (done = 1).
__global__ void __launch_bounds__(LIN_NODE_THREADS) k_lin_direction(LinArgs A) {
    __shared__ bool last_sh;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    CgCtl* ctl = A.ctl;
    const int done = __ldcg(&ctl->done);
    if (done == 1) return;
    const double alpha = __ldcg(&ctl->alpha), beta = __ldcg(&ctl->beta);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.N) {
        const size_t k = 3 * (size_t)i;
        const double rv[3] = {A.r[k], A.r[k + 1], A.r[k + 2]}, uv[3] = {A.u[k], A.u[k + 1], A.u[k + 2]};
        double* pi = A.p + 4 * (size_t)i;
        double pv[3];
        ld_node(pi, pv);
#pragma unroll
        for (int d = 0; d < 3; ++d) A.u[k + d] = uv[d] + alpha * pv[d];
        if (done == 0) st_node(pi, rv[0] + beta * pv[0], rv[1] + beta * pv[1], rv[2] + beta * pv[2]);
    }
    if (done == 2) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            last_sh = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
            if (last_sh) {
                ctl->ticket = 0u;
                ctl->done = 1;
            }
        }
    }
}

// p = r = f, u = 0, r.r.
__global__ void __launch_bounds__(LIN_NODE_THREADS) k_lin_init(LinArgs A) {
    __shared__ double red[LIN_NODE_THREADS / 32];
    __shared__ bool last_sh;
    CgCtl* ctl = A.ctl;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    if (i < A.N) {
        const size_t k = 3 * (size_t)i;
        const double fv[3] = {A.f[k], A.f[k + 1], A.f[k + 2]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            A.u[k + d] = 0.0;
            A.r[k + d] = fv[d];
            s += fv[d] * fv[d];
        }
        st_node(A.p + 4 * (size_t)i, fv[0], fv[1], fv[2]);
    }
    double rr;
    if (lin_last_fold(s, A.part, (int)gridDim.x, &ctl->ticket, red, &last_sh, &rr) && threadIdx.x == 0) {
        ctl->rr0 = ctl->rr = rr;
        ctl->rel = 1.0;
        if (rr == 0.0) {
            ctl->done = 1;
            ctl->rel = 0.0;
        } else if (A.max_iter <= 0) {
            ctl->done = 1;
            ctl->status = 2;
        }
    }
}

// Apply: x with the eliminated DOFs dropped, and y = K x with their identity rows.
__global__ void k_lin_mask(LinArgs A, const double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.N) return;
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = A.is_fixed[3 * (size_t)i + d] ? 0.0 : x[3 * (size_t)i + d];
    st_node(A.p + 4 * (size_t)i, v[0], v[1], v[2]);
}

__global__ void k_lin_collect(LinArgs A, const double* __restrict__ x, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.N) return;
    double q[3];
    lin_node_sum(A.slots, A.node_soff[i], A.node_soff[i + 1], q);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const size_t k = 3 * (size_t)i + d;
        y[k] = A.is_fixed[k] ? x[k] : q[d];
    }
}

}  // namespace tlfea

// batch_lin.cuh -- the phases of the batched CG on straight-sided elements (straight.cuh): the
// element tiles as lin_cg.cuh's pipelined product, p and the tile sums in 32-byte node records,
// and an iteration of three phases instead of five launches:
//
//   tiles       K p per tile into the node slots, and each (tile, instance) pair's share of
//               p.Kp; one pass of a tile's tables and geometry serves a group of instances
//               when the mesh is shared;
//   update      alpha = rr / p.Kp folded by every warp from its instance's pairs (no ticket),
//               r -= alpha q per node chunk, r.r per chunk;
//   direction   r.r folded the same way, the stop test, u += alpha p, p = r + beta p.
//
// One block per node chunk in the last two (a warp per chunk left 7 warps per SM on 48 beams of
// 260,000 nodes: 27 us for the update); the first chunk of an instance writes its
// scalars.  An instance that ends in iteration it is stamped it + 1 and counts as done from the
// next one, so the warps of one phase agree whatever their order.
#pragma once

#include "force_pipe.cuh"
#include "straight.cuh"

namespace tlfea {

constexpr int BL_RUNNING = 0x7fffffff;  // stamp of a running instance

template <typename R>
struct BLinArgs {
    const int* node_off;
    const int* pad_off;
    const int* pad_gid;
    const int* pad_slot;
    const uint16_t* pad_iend;
    const uint16_t* inc;
    const uint16_t* lconn;
    const R* geo;
    const int* node_soff;
    const R* lam;  // per element slot; shared mesh: per instance
    const R* mu;
    int n_tiles, max_local;
    int group;  // shared mesh: instances per pass of a tile's tables
    // shared mesh: nodes and node slots per instance (0 otherwise)
    int nodes_per_inst, slots_per_inst;
    int N, n_inst, n_chunks;
    const unsigned char* fixed;  // per node
    const int* chunk_inst;
    const int* chunk_beg;
    const int* inst_chunk;
    const int* tile_inst;  // first and last instance of a tile (not for a shared mesh)
    const int* tile_pair;  // first (tile, instance) pair of a tile
    const int* inst_pair;  // first pair of an instance: its pairs are contiguous
    const int* node_inst;
    double *u, *r;
    double* p;      // 4 per node
    double* slots;  // 4 per node slot
    double* pair;   // p.Kp per (tile, instance)
    double *cpa, *cpb, *rr, *fnorm, *rel, *alpha;
    const double* f;
    const double* u0;
    int *iters, *status, *done, *n_done, *stamp, *flag;
    LinRule rule;
    int* err;
};

// Shared memory: [element forces][p][local connectivity][the scatter's tables twice][barriers: the
// tables', the connectivity's].  The connectivity is read before the scatter starts, so one copy
// is refilled meanwhile; the fourth block per SM needs the room.
template <typename R, int NPE>
struct BLinLayout {
    size_t p, lconn, tab, inc, slot, iend, tab_bytes, bar, total;
    __host__ __device__ explicit BLinLayout(int ml) {
        auto al = [](size_t v) { return (v + 15) & ~size_t(15); };
        p = al(3 * (size_t)NPE * TILE_ELEMS * sizeof(R));
        lconn = al(p + 3 * (size_t)ml * sizeof(double));
        tab = lconn + NPE * TILE_ELEMS * sizeof(uint16_t);
        inc = 0;
        slot = inc + NPE * TILE_ELEMS * sizeof(uint16_t);
        iend = slot + (size_t)ml * sizeof(int);
        tab_bytes = al(iend + (size_t)ml * sizeof(uint16_t));
        bar = tab + 2 * tab_bytes;
        total = bar + 24;
    }
};


__device__ __forceinline__ void bl_init_barriers(uint32_t bar) {
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
        mbar_init(bar + 16, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
}

// K p over the tiles of the instances that are running in iteration `it` (skip = false: of
// all).  `loads` counts the table loads of this block since bl_init_barriers; -1 from the first
// table on that did not land: the block does no more products.  The work of a
// block is a sequence of units (item, instance); the next unit's p (and, where the tile
// changes, its tables and geometry) are in flight while the current one is computed.
template <typename R, int NPE, bool SH>
__device__ __forceinline__ void bl_tiles(const BLinArgs<R>& A, int it, bool skip, unsigned char* smem, int& loads) {
    constexpr int TE = TILE_ELEMS, NB = 3;
    __shared__ double red[TE / 32];
    const int t = threadIdx.x;
    const BLinLayout<R, NPE> L(A.max_local);
    R* fe = reinterpret_cast<R*>(smem);
    double* ps = reinterpret_cast<double*>(smem + L.p);
    const uint32_t bar0 = smem_u32(smem + L.bar);
    const int groups = SH ? (A.n_inst + A.group - 1) / A.group : 1;
    const int n_items = A.n_tiles * groups;
    auto running = [&](int b) { return !skip || __ldcg(A.stamp + b) > it; };
    // the first unit at or after (item, inst); item = n_items: none
    auto seek = [&](int& item, int& inst) {
        for (; item < n_items; item += gridDim.x) {
            if constexpr (SH) {  // a lane per instance of the group (up to eight): one round trip
                const int g0 = (item / A.n_tiles) * A.group, b = g0 + (t & 31);
                const bool run = (t & 31) < A.group && b >= inst && b < A.n_inst && running(b);
                if (const unsigned m = __ballot_sync(0xffffffffu, run)) {
                    inst = g0 + __ffs(m) - 1;
                    return;
                }
                inst = 0;
            } else {
                for (int b = A.tile_inst[2 * item]; b <= A.tile_inst[2 * item + 1]; ++b)
                    if (running(b)) return;
            }
        }
        item = n_items;
    };
    auto issue = [&](int tile, int load) {  // thread 0
        constexpr uint32_t TAB = NPE * TE * sizeof(uint16_t);
        const uint32_t bar = bar0 + 8 * (load & 1);
        unsigned char* tab = smem + L.tab + (load & 1) * L.tab_bytes;
        const int pb = A.pad_off[tile];
        const uint32_t np = (uint32_t)(A.pad_off[tile + 1] - pb);
        mbar_expect_tx(bar, TAB + np * (sizeof(int) + sizeof(uint16_t)));
        bulk_g2s(smem_u32(tab + L.inc), A.inc + (size_t)tile * NPE * TE, TAB, bar);
        bulk_g2s(smem_u32(tab + L.slot), A.pad_slot + pb, np * sizeof(int), bar);
        bulk_g2s(smem_u32(tab + L.iend), A.pad_iend + pb, np * sizeof(uint16_t), bar);
    };
    auto issue_lconn = [&](int tile) {  // thread 0
        constexpr uint32_t TAB = NPE * TE * sizeof(uint16_t);
        mbar_expect_tx(bar0 + 16, TAB);
        bulk_g2s(smem_u32(smem + L.lconn), A.lconn + (size_t)tile * NPE * TE, TAB, bar0 + 16);
    };
    R ji[9], det, lam, mu;
    double pv[NB][3];
    auto geometry = [&](int tile) {
        const R* g = A.geo + (size_t)tile * 10 * TE + t;
#pragma unroll
        for (int m = 0; m < 9; ++m) ji[m] = __ldg(g + m * TE);
        det = __ldg(g + 9 * TE);
        if constexpr (!SH) {
            lam = __ldg(A.lam + (size_t)tile * TE + t);
            mu = __ldg(A.mu + (size_t)tile * TE + t);
        }
    };
    auto gather = [&](int tile, int inst, int n) {
        const int pb = A.pad_off[tile];
        int g[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) g[j] = A.pad_gid[pb + min(t + j * TE, n - 1)];
        const double* p = A.p + (SH ? 4 * (size_t)inst * A.nodes_per_inst : 0);
#pragma unroll
        for (int j = 0; j < NB; ++j) ld_node_shared(p + 4 * (size_t)g[j], pv[j]);
    };
    int item = blockIdx.x, inst = 0;
    seek(item, inst);
    if (item >= n_items || loads < 0) return;
    int tile = item % A.n_tiles;
    int nl = A.node_off[tile + 1] - A.node_off[tile];
    if (t == 0) {
        issue(tile, loads);
        issue_lconn(tile);
    }
    geometry(tile);
    gather(tile, inst, nl);
    bool fresh = true;  // this unit's tables are still on their way
    while (item < n_items) {
        const int load = loads;
        const bool landed =
            !fresh || (mbar_wait(bar0 + 8 * (load & 1), (load >> 1) & 1) && mbar_wait(bar0 + 16, load & 1));
        const unsigned char* tab = smem + L.tab + (load & 1) * L.tab_bytes;
        const uint16_t* incs = reinterpret_cast<const uint16_t*>(tab + L.inc);
        const uint16_t* lcs = reinterpret_cast<const uint16_t*>(smem + L.lconn);
        const int* slot = reinterpret_cast<const int*>(tab + L.slot);
        const uint16_t* iends = reinterpret_cast<const uint16_t*>(tab + L.iend);
        if constexpr (SH) {
            lam = __ldg(A.lam + inst);
            mu = __ldg(A.mu + inst);
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int ln = t + j * TE;
            if (ln < nl) {
#pragma unroll
                for (int d = 0; d < 3; ++d) ps[3 * ln + d] = pv[j][d];
            }
        }
        for (int ln = t + NB * TE; ln < nl; ln += TE) {  // larger tiles
            ld_node_shared(A.p + (SH ? 4 * (size_t)inst * A.nodes_per_inst : 0) +
                               4 * (size_t)A.pad_gid[A.pad_off[tile] + ln],
                           pv[0]);
#pragma unroll
            for (int d = 0; d < 3; ++d) ps[3 * ln + d] = pv[0][d];
        }
        int item2 = item, inst2 = inst + 1;
        if constexpr (!SH) item2 += gridDim.x;
        seek(item2, inst2);
        const bool more = item2 < n_items;
        const int tile2 = more ? item2 % A.n_tiles : tile;
        const bool swap = more && item2 != item;
        // p staged; the other table buffer's readers are past it
        if (!__syncthreads_and(landed)) {
            tables_late(A.err, bar0 + 8 * (load & 1), (load >> 1) & 1);
            mbar_wait(bar0 + 16, load & 1);
            loads = -1;
            return;
        }
        if (swap && t == 0) issue(tile2, load + 1);
        {
            int lc[NPE];
#pragma unroll
            for (int a = 0; a < NPE; ++a) lc[a] = 3 * lcs[a * TE + t];
            lin_element<R, NPE>(ji, det, lam, mu, A.rule, [&](int a, int c) { return ps[lc[a] + c]; }, fe + t);
        }
        const int nl_now = nl;
        if (more) {  // in flight during the scatter
            if (swap) {
                nl = A.node_off[tile2 + 1] - A.node_off[tile2];
                geometry(tile2);
            }
            gather(tile2, inst2, nl);
        }
        if (swap) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // reads of lconn before its refill
        __syncthreads();  // element forces complete
        if (swap && t == 0) issue_lconn(tile2);
        double dot = 0.0;
        double* slots = A.slots + (SH ? 4 * (size_t)inst * A.slots_per_inst : 0);
        const int lo = SH ? inst : A.tile_inst[2 * tile], hi = SH ? inst : A.tile_inst[2 * tile + 1];
        for (int ln = t; ln < nl_now; ln += TE) {
            double s0, s1, s2;
            tile_node_sum(fe, incs, ln ? iends[ln - 1] : 0, iends[ln], s0, s1, s2);
            st_node(slots + 4 * (size_t)slot[ln], s0, s1, s2);
            const double d = ps[3 * ln + 0] * s0 + ps[3 * ln + 1] * s1 + ps[3 * ln + 2] * s2;
            if (lo != hi) ps[3 * ln] = d;  // (this thread alone reads ps[ln] by now)
            dot += d;
        }
        for (int b = lo; b <= hi; ++b) {  // one pass, unless the tile holds several instances
            if (lo != hi) {
                dot = 0.0;
                for (int ln = t; ln < nl_now; ln += TE)
                    if (A.node_inst[A.pad_gid[A.pad_off[tile] + ln]] == b) dot += ps[3 * ln];
                __syncthreads();  // red free
            }
            const double w = warp_sum(dot);
            if ((t & 31) == 0) red[t >> 5] = w;
            // every thread's reads of the tables precede the bulk copies that replace them
            if (b == hi) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();  // sums posted; after the last pass fe, ps and the tables are free
            if (t == 0)
                A.pair[SH ? inst * A.n_tiles + tile : A.tile_pair[tile] + (b - lo)] =
                    (red[0] + red[1]) + (red[2] + red[3]);
        }
        fresh = swap;
        if (swap) ++loads;
        item = item2;
        inst = inst2;
        tile = tile2;
    }
    ++loads;  // the last tables were consumed
}

// q = K p of node i of instance b: the node's slots in tile order, two in flight.
template <typename R>
__device__ __forceinline__ void bl_node_sum(const BLinArgs<R>& A, int i, int b, double q[3]) {
    const int l = A.nodes_per_inst ? i - b * A.nodes_per_inst : i;
    const double* slots = A.slots + 4 * (size_t)b * A.slots_per_inst;
    const int so = A.node_soff[l], se = A.node_soff[l + 1];
    q[0] = q[1] = q[2] = 0.0;
    for (int k = so; k < se; k += 2) {
        double v[2][3];
        ld_node_shared(slots + 4 * (size_t)k, v[0]);
        ld_node_shared(slots + 4 * (size_t)min(k + 1, se - 1), v[1]);
#pragma unroll
        for (int d = 0; d < 3; ++d) q[d] += v[0][d];
        if (k + 1 < se) {
#pragma unroll
            for (int d = 0; d < 3; ++d) q[d] += v[1][d];
        }
    }
}

// Sum of [b, e) by one warp, in every lane.
__device__ __forceinline__ double bl_fold(const double* v, int b, int e) {
    double s = 0.0;
    for (int k = b + (threadIdx.x & 31); k < e; k += 32) s += __ldcg(v + k);
    return warp_sum(s);
}

// Sum over the block (warps in order), in thread 0; called by all its threads.
__device__ __forceinline__ double bl_block_sum(double v) {
    __shared__ double red[TILE_ELEMS / 32];
    v = warp_sum(v);
    __syncthreads();  // red free
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    return (red[0] + red[1]) + (red[2] + red[3]);
}

// u = p = u0 (warm) or 0, r = f_free; ||f_free||^2 per chunk.
template <typename R>
__device__ __forceinline__ void bl_start(const BLinArgs<R>& A, int warm) {
    const int t = threadIdx.x;
    for (int c = blockIdx.x; c < A.n_chunks; c += gridDim.x) {
        double s = 0.0;
        for (int i = A.chunk_beg[c] + t; i < A.chunk_beg[c + 1]; i += TILE_ELEMS) {
            const bool fx = A.fixed[i];
            double uv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const size_t k = 3 * (size_t)i + d;
                const double fv = fx ? 0.0 : A.f[k];
                uv[d] = (warm && !fx) ? A.u0[k] : 0.0;
                A.r[k] = fv;
                A.u[k] = uv[d];
                s += fv * fv;
            }
            st_node(A.p + 4 * (size_t)i, uv[0], uv[1], uv[2]);
        }
        s = bl_block_sum(s);
        if (t == 0) A.cpa[c] = s;
    }
}

// r -= K u0 (warm), p = r; ||r||^2 per chunk.
template <typename R>
__device__ __forceinline__ void bl_residual(const BLinArgs<R>& A, int warm) {
    const int t = threadIdx.x;
    for (int c = blockIdx.x; c < A.n_chunks; c += gridDim.x) {
        const int b = A.chunk_inst[c];
        double s = 0.0;
        for (int i = A.chunk_beg[c] + t; i < A.chunk_beg[c + 1]; i += TILE_ELEMS) {
            double q[3] = {0.0, 0.0, 0.0}, rv[3];
            if (warm && !A.fixed[i]) bl_node_sum(A, i, b, q);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                rv[d] = A.r[3 * (size_t)i + d] - q[d];
                A.r[3 * (size_t)i + d] = rv[d];
                s += rv[d] * rv[d];
            }
            st_node(A.p + 4 * (size_t)i, rv[0], rv[1], rv[2]);
        }
        s = bl_block_sum(s);
        if (t == 0) A.cpb[c] = s;
    }
}

// Per instance, one warp each: ||f_free||, rr_0, the initial relative residual and state.
template <typename R>
__device__ __forceinline__ void bl_init(const BLinArgs<R>& A, double tol) {
    const int warps = blockDim.x / 32;
    for (int b = blockIdx.x * warps + (threadIdx.x >> 5); b < A.n_inst; b += gridDim.x * warps) {
        const double fn = sqrt(bl_fold(A.cpa, A.inst_chunk[b], A.inst_chunk[b + 1]));
        const double rr0 = bl_fold(A.cpb, A.inst_chunk[b], A.inst_chunk[b + 1]);
        if ((threadIdx.x & 31) == 0) {
            const double rel = (fn > 0.0) ? sqrt(rr0) / fn : 0.0;
            const bool dn = fn == 0.0 || rel < tol;
            A.fnorm[b] = fn;
            A.rr[b] = rr0;
            A.rel[b] = rel;
            A.iters[b] = 0;
            A.status[b] = 0;
            A.flag[b] = 0;
            A.stamp[b] = dn ? -1 : BL_RUNNING;
            if (dn) atomicAdd(A.n_done, 1);
        }
    }
}

// f(c, b) for the block's chunks c whose instance b runs in iteration `it`.  A lane looks at a
// chunk: a large batch of which few instances are left would spend its time on blocks and round
// trips that find nothing to do.
template <typename R, typename F>
__device__ __forceinline__ void bl_running_chunks(const BLinArgs<R>& A, int it, F f) {
    for (long long c0 = blockIdx.x; c0 < A.n_chunks; c0 += 32LL * gridDim.x) {
        const long long c = c0 + (long long)(threadIdx.x & 31) * gridDim.x;
        const int b = c < A.n_chunks ? A.chunk_inst[c] : 0;
        unsigned m = __ballot_sync(0xffffffffu, c < A.n_chunks && __ldcg(A.stamp + b) > it);
        for (; m; m &= m - 1) {  // uniform over the block: a stamp set in this phase is above `it`
            const int k = __ffs(m) - 1;
            f((int)(c0 + (long long)k * gridDim.x), __shfl_sync(0xffffffffu, b, k));
        }
    }
}

// alpha, r -= alpha q, r.r per chunk.
template <typename R>
__device__ __forceinline__ void bl_update(const BLinArgs<R>& A, int it) {
    const int t = threadIdx.x;
    const double* rr_old = A.rr + (size_t)(it & 1) * A.n_inst;
    bl_running_chunks(A, it, [&](int c, int b) {
        const bool first = t == 0 && c == A.inst_chunk[b];
        const double pq = bl_fold(A.pair, A.inst_pair[b], A.inst_pair[b + 1]);
        if (!(pq > 0.0)) {  // non-positive p.Kp: the reference aborts this solve
            if (first) {
                A.flag[b] = 2;
                A.status[b] = 1;
                A.stamp[b] = it + 1;
                atomicAdd(A.n_done, 1);
            }
            return;
        }
        const double alpha = __ldcg(rr_old + b) / pq;
        if (first) A.alpha[b] = alpha;
        const int i_end = A.chunk_beg[c + 1];
        double s = 0.0;
        for (int i0 = A.chunk_beg[c] + t; i0 < i_end; i0 += 2 * TILE_ELEMS) {
            double rv[2][3], q[2][3];
            bool ok[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int i = min(i0 + TILE_ELEMS * j, i_end - 1);
                ok[j] = i0 + TILE_ELEMS * j < i_end && !A.fixed[i];
#pragma unroll
                for (int d = 0; d < 3; ++d) rv[j][d] = __ldcg(A.r + 3 * (size_t)i + d);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) bl_node_sum(A, min(i0 + TILE_ELEMS * j, i_end - 1), b, q[j]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (!ok[j]) continue;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double ri = rv[j][d] - alpha * q[j][d];
                    A.r[3 * (size_t)(i0 + TILE_ELEMS * j) + d] = ri;
                    s += ri * ri;
                }
            }
        }
        s = bl_block_sum(s);
        if (t == 0) A.cpb[c] = s;
    });
}

// The stop test and beta, u += alpha p, p = r + beta p.
template <typename R>
__device__ __forceinline__ void bl_direction(const BLinArgs<R>& A, int it, double tol, int max_iter) {
    const int t = threadIdx.x;
    const double* rr_old = A.rr + (size_t)(it & 1) * A.n_inst;
    bl_running_chunks(A, it, [&](int c, int b) {
        if (__ldcg(A.flag + b) == 2) return;
        const double alpha = __ldcg(A.alpha + b);
        const double rrn = bl_fold(A.cpb, A.inst_chunk[b], A.inst_chunk[b + 1]);
        const double rel = sqrt(rrn) / __ldcg(A.fnorm + b);
        const bool conv = rel < tol;
        const double beta = rrn / __ldcg(rr_old + b);
        if (t == 0 && c == A.inst_chunk[b]) {
            A.rr[(size_t)((it + 1) & 1) * A.n_inst + b] = rrn;
            A.iters[b] = it + 1;
            A.rel[b] = rel;
            if (conv) {
                A.stamp[b] = it + 1;
                atomicAdd(A.n_done, 1);
            } else if (it + 1 >= max_iter) {
                A.status[b] = 2;
            }
        }
        const int i_end = A.chunk_beg[c + 1];
        for (int i0 = A.chunk_beg[c] + t; i0 < i_end; i0 += 2 * TILE_ELEMS) {
            double rv[2][3], uv[2][3], pv[2][3];
#pragma unroll
            for (int j = 0; j < 2; ++j) {  // every load before the first store
                const int i = min(i0 + TILE_ELEMS * j, i_end - 1);
                ld_node_shared(A.p + 4 * (size_t)i, pv[j]);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    rv[j][d] = __ldcg(A.r + 3 * (size_t)i + d);
                    uv[j][d] = __ldcg(A.u + 3 * (size_t)i + d);
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int i = i0 + TILE_ELEMS * j;
                if (i >= i_end) continue;
#pragma unroll
                for (int d = 0; d < 3; ++d) A.u[3 * (size_t)i + d] = uv[j][d] + alpha * pv[j][d];
                if (!conv)
                    st_node(A.p + 4 * (size_t)i, rv[j][0] + beta * pv[j][0], rv[j][1] + beta * pv[j][1],
                            rv[j][2] + beta * pv[j][2]);
            }
        }
    });
}

// Instances still running at the iteration cap end with status 2; the done flags.
template <typename R>
__device__ __forceinline__ void bl_finish(const BLinArgs<R>& A) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < A.n_inst; b += gridDim.x * blockDim.x) {
        const bool run = A.stamp[b] == BL_RUNNING;
        A.done[b] = run ? 0 : 1;
        if (run && A.status[b] == 0) A.status[b] = 2;
    }
}

// Products are missing: every instance counts as ended (called where n_done may grow; the host
// reads the error word).
template <typename R>
__device__ __forceinline__ void bl_end_if_late(const BLinArgs<R>& A, int loads) {
    if (loads < 0 && threadIdx.x == 0) atomicMax(A.n_done, A.n_inst);
}

// ---- one launch per phase (mode 0).  Iteration j of a captured chunk is *base + j; a phase
// past the cap, or that finds every instance done, returns.  n_done only grows in the phases
// after their own test of it matters (an instance that ends in the direction phase still gets
// its u there: that phase goes by the stamps).
__device__ __forceinline__ void bl_enter() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename R, int NPE, bool SH>
__global__ void __launch_bounds__(TILE_ELEMS, 4) k_bl_tiles(BLinArgs<R> A, const int* base, int j, int skip,
                                                            int max_iter) {
    extern __shared__ __align__(128) unsigned char smem[];
    bl_enter();
    const int it = skip ? __ldcg(base) + j : 0;
    if (skip && (it >= max_iter || __ldcg(A.n_done) >= A.n_inst)) return;
    bl_init_barriers(smem_u32(smem + BLinLayout<R, NPE>(A.max_local).bar));
    int loads = 0;
    bl_tiles<R, NPE, SH>(A, it, skip != 0, smem, loads);
    if (skip) bl_end_if_late(A, loads);
}
template <typename R>
__global__ void __launch_bounds__(TILE_ELEMS) k_bl_start(BLinArgs<R> A, int warm) {
    bl_start(A, warm);
}
template <typename R>
__global__ void __launch_bounds__(TILE_ELEMS) k_bl_residual(BLinArgs<R> A, int warm) {
    bl_residual(A, warm);
}
template <typename R>
__global__ void __launch_bounds__(TILE_ELEMS) k_bl_init(BLinArgs<R> A, double tol) {
    bl_init(A, tol);
}
template <typename R>
__global__ void __launch_bounds__(TILE_ELEMS) k_bl_update(BLinArgs<R> A, const int* base, int j, int max_iter) {
    bl_enter();
    const int it = __ldcg(base) + j;
    if (it >= max_iter) return;
    bl_update(A, it);
}
template <typename R>
__global__ void __launch_bounds__(TILE_ELEMS) k_bl_direction(BLinArgs<R> A, const int* base, int j, double tol,
                                                             int max_iter) {
    bl_enter();
    const int it = __ldcg(base) + j;
    if (it >= max_iter) return;
    bl_direction(A, it, tol, max_iter);
}
__global__ void k_bl_advance(int* base, int n) {
    bl_enter();
    *base += n;
}
template <typename R>
__global__ void k_bl_finish(BLinArgs<R> A) {
    bl_finish(A);
}

// Apply, the solve's own product: p = x with the fixed nodes' columns dropped, and y = K x with
// their identity rows.
template <typename R>
__global__ void k_bl_mask(BLinArgs<R> A, const double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.N) return;
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = A.fixed[i] ? 0.0 : x[3 * (size_t)i + d];
    st_node(A.p + 4 * (size_t)i, v[0], v[1], v[2]);
}
template <typename R>
__global__ void k_bl_collect(BLinArgs<R> A, const double* __restrict__ x, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.N) return;
    double q[3];
    bl_node_sum(A, i, A.nodes_per_inst ? i / A.nodes_per_inst : 0, q);
#pragma unroll
    for (int d = 0; d < 3; ++d) y[3 * (size_t)i + d] = A.fixed[i] ? x[3 * (size_t)i + d] : q[d];
}

// ---- the whole solve in one cooperative launch (mode 1): the same phases.
template <typename R, int NPE, bool SH>
__global__ void __launch_bounds__(TILE_ELEMS, 4) k_bl_cg(BLinArgs<R> A, double tol, int max_iter, int warm) {
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    extern __shared__ __align__(128) unsigned char smem[];
    bl_init_barriers(smem_u32(smem + BLinLayout<R, NPE>(A.max_local).bar));
    int loads = 0;
    bl_start(A, warm);
    grid.sync();
    if (warm) {
        bl_tiles<R, NPE, SH>(A, 0, false, smem, loads);
        grid.sync();
    }
    bl_residual(A, warm);
    grid.sync();
    bl_init(A, tol);
    bl_end_if_late(A, loads);
    grid.sync();
    for (int it = 0; it < max_iter; ++it) {
        if (__ldcg(A.n_done) >= A.n_inst) break;  // uniform: read after a grid barrier, grows before one
        bl_tiles<R, NPE, SH>(A, it, true, smem, loads);
        grid.sync();
        bl_update(A, it);
        grid.sync();
        bl_direction(A, it, tol, max_iter);
        bl_end_if_late(A, loads);
        grid.sync();
    }
    bl_finish(A);
}

}  // namespace tlfea

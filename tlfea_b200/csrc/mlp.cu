// mlp.cu -- the warm-start network: a small MLP (dims[0] -> ... -> dims[L],
// GELU between layers) trained and evaluated on the GPU by this file's own
// kernels.  New, no reference counterpart.
//
// Every matrix product is one tcgen05 kernel (k_gemm_bf16<BN>):
//     D[M x N] (FP32) = A[M x K] (BF16) * B[N x K]^T (BF16) (+ bias[N])
// with both operands K-major (row-major with K contiguous).  A CTA owns a
// 128-row x BN-column tile (BN = 64, 128 or 256, chosen per product so that
// small products still spread over many SMs).  K streams through a ring of
// GM_STAGES shared-memory stages, 64 elements (one 128-byte row) at a time:
// one thread issues two tiled tensor copies per stage (A's 128 x 64 box and
// B's BN x 64 box, 128-byte swizzle, rows past M / N and columns past K read
// as zero), waits for the stage, issues four tcgen05.mma (kind::f16, BF16 in,
// FP32 accumulator in TMEM) and commits them to the stage's "empty" barrier;
// the stage is refilled as soon as the products that read it have finished,
// so the copies of the next stages overlap the tensor-core work.  The four
// warps then read the accumulator back with tcgen05.ld (warp w owns TMEM
// lanes 32w..32w+31) and store D.
//
// Training keeps FP32 master weights and BF16 copies in both layouts
// (W [N x Kp] for the forward product, W^T [Kp x N] for the input gradient),
// and writes activations and output gradients in both layouts too, so every
// product -- forward, input gradient, weight gradient -- is the same K-major
// kernel.  The optimiser is AdamW.  Reductions (bias gradients, the loss) are
// fixed-order, so a training run is deterministic.
//
// A training step of L layers is 2 L + 2 launches: the input's layouts, L forward products whose
// epilogues add the bias and apply GELU (the last forms the loss and its gradient), L - 1 launches
// of an input gradient beside its layer's weight gradient, the first layer's weight gradient, and
// the bias sums with the whole AdamW step.  At batch 512 with three hidden layers of 256 and 64
// outputs every product is a few microseconds on 2 to 16 CTAs, so the step is a chain of launches
// and of first reads; it took 285 us with separate activation, loss, bias and optimiser kernels and a
// host-side tensor-map encode per product, 176 us with those in the products' epilogues, 80 us
// with 512-thread epilogues, the paired gradients and one coalesced AdamW launch (in the weight
// gradient's epilogue the optimiser ran on 2 to 8 CTAs, 22 to 31 us each).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "force_pipe.cuh"

namespace tlfea {

constexpr int MLP_TM = 128;    // rows per CTA (the MMA's M)
constexpr int GM_BK = 64;      // K elements per stage: one 128-byte swizzle row
constexpr int GM_STAGES = 4;   // shared-memory ring depth
constexpr int GM_GROUP = 16;   // row tiles per group of the tile order

template <int BN>
struct GemmGeom {
    static constexpr uint32_t A_BYTES = MLP_TM * GM_BK * 2;
    static constexpr uint32_t B_BYTES = BN * GM_BK * 2;
    static constexpr uint32_t STAGE = A_BYTES + B_BYTES;  // a multiple of 1024 (swizzle atoms stay aligned)
    static constexpr size_t SMEM = 1024 + (size_t)GM_STAGES * STAGE;  // + slack to align the ring to 1024 B
};

struct GemmArgs {
    int M, N, K;
    const __nv_bfloat16* A;
    int lda;
    const __nv_bfloat16* B;
    int ldb;
    const float* bias;
    float* D;
    int ldd;
    int* err;
};

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzle
// layout that the tensor copies write: rows of 128 bytes, 8-row groups 1024
// bytes apart (stride byte offset), descriptor version 1, swizzle mode 2
// (128 bytes).  The leading byte offset is unused for this layout.  A K step
// of 16 elements inside the 128-byte row advances the start address by 32 B.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Tiled 2-D tensor copy global -> shared (box given by the tensor map), completion
// counted on `bar`; x is the K coordinate (a multiple of 64 here, so 128-byte aligned).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// One tile of a product with an epilogue: epi(row, col, v, live) gets 16 consecutive columns of a
// row of the accumulator (live: row < M; every lane of a warp calls it), epi.finish(tile) runs
// once per thread after the CTA's last of them.  NT threads: every four warps take the next 16
// columns (a warp reads the TMEM lanes of its quarter).  The network's epilogues do real work per
// element on few CTAs (16 for 512 x 256), so they run 512 threads, a chunk of 16 columns each at
// BN = 64.
template <int BN, int NT, typename Epi>
__device__ __forceinline__ void gemm_tile(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int tile,
                                          Epi& epi) {
    using G = GemmGeom<BN>;
    extern __shared__ unsigned char gemm_smem[];
    __shared__ __align__(8) unsigned long long bars[2 * GM_STAGES + 1];  // full[S], empty[S], done
    __shared__ uint32_t tmem_sh;
    __shared__ int ok_sh;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // grouped tile order: consecutive CTAs walk GM_GROUP row tiles down one
    // column tile before moving right, so the CTAs resident at one time share a
    // few A row panels and B column panels in L2
    const int mtiles = (g.M + MLP_TM - 1) / MLP_TM, ntiles = (g.N + BN - 1) / BN;
    const int per_group = GM_GROUP * ntiles, grp = tile / per_group;
    const int first_m = grp * GM_GROUP, gm = min(mtiles - first_m, GM_GROUP);
    const int in_grp = tile - grp * per_group;
    const int m0 = (first_m + in_grp % gm) * MLP_TM, n0 = (in_grp / gm) * BN;
    const int nk = (g.K + GM_BK - 1) / GM_BK;
    const uint32_t ring = (smem_u32(gemm_smem) + 1023u) & ~1023u;
    const uint32_t bar0 = smem_u32(bars), done = bar0 + 16 * GM_STAGES;
    auto full = [&](int s) { return bar0 + 8 * s; };
    auto empty = [&](int s) { return bar0 + 8 * (GM_STAGES + s); };
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "n"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (t == 0) {
        for (int i = 0; i < 2 * GM_STAGES + 1; ++i) mbar_init(bar0 + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tb)) : "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    // (a programmatic dependent of its predecessor, where it was launched as one)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == 0) {
        if (lane == 0) {
            // one thread: copies into the ring and tensor-core issue
            constexpr uint32_t idesc = umma_idesc_bf16(MLP_TM, BN);
            bool ok = true;
            int loaded = 0, landed = 0;
            auto load = [&](int k) {
                const int s = k % GM_STAGES;
                const uint32_t a = ring + s * G::STAGE;
                mbar_expect_tx(full(s), G::STAGE);
                tma_load_2d(a, &ta, k * GM_BK, m0, full(s));
                tma_load_2d(a + G::A_BYTES, &tb, k * GM_BK, n0, full(s));
            };
            for (; loaded < nk && loaded < GM_STAGES; ++loaded) load(loaded);
            for (int k = 0; k < nk; ++k) {
                const int s = k % GM_STAGES;
                if (!mbar_wait(full(s), (k / GM_STAGES) & 1)) {
                    ok = false;
                    break;
                }
                landed = k + 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = ring + s * G::STAGE, b = a + G::A_BYTES;
#pragma unroll
                for (int kk = 0; kk < GM_BK / 16; ++kk) {
                    const uint64_t ad = umma_desc_sw128(a + 32 * kk), bd = umma_desc_sw128(b + 32 * kk);
                    const uint32_t acc = (k > 0 || kk > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                        : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 empty(s))
                             : "memory");
                // refill the stage that the previous chunk's products read (they have
                // had this chunk's issue time to finish; the tensor pipe keeps a queue)
                if (k >= 1 && loaded < nk) {
                    const int sp = (k - 1) % GM_STAGES;
                    if (!mbar_wait(empty(sp), ((k - 1) / GM_STAGES) & 1)) {
                        ok = false;
                        break;
                    }
                    load(loaded++);
                }
            }
            // arrives once every product issued above has completed
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(done)
                         : "memory");
            if (!ok) {
                atomicExch(g.err, 5);
                // copies still in flight land before the CTA's shared memory is released
                for (int k = landed; k < loaded; ++k) mbar_wait(full(k % GM_STAGES), (k / GM_STAGES) & 1);
            }
            ok_sh = ok ? 1 : 0;
        }
        __syncwarp();
    }
    const bool got = mbar_wait(done, 0);
    const bool ok = __syncthreads_and(got) && ok_sh;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        const int quarter = warp & 3, row = m0 + quarter * 32 + lane;
        const int ncols = min(BN, g.N - n0);
        for (int c0 = (warp >> 2) * 16; c0 < ncols; c0 += NT / 8) {
            uint32_t v[16];
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                "%13, %14, %15}, [%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(taddr)
                : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            epi(row, n0 + c0, v, row < g.M);  // N is a multiple of 16, so every chunk is whole
        }
        epi.finish(tile);
    } else if (t == 0) {
        atomicExch(g.err, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(BN) : "memory");
}

template <int BN, int NT, typename Epi>
__global__ void __launch_bounds__(NT) k_gemm_bf16(const __grid_constant__ CUtensorMap ta,
                                                  const __grid_constant__ CUtensorMap tb, GemmArgs g, Epi epi) {
    asm volatile("griddepcontrol.launch_dependents;");
    gemm_tile<BN, NT>(ta, tb, g, blockIdx.x, epi);
}

// Two independent products in one launch, the first on the first `tiles` CTAs: a layer's input
// gradient, which the next launch waits for, beside its weight gradient, which nothing does.
template <int BN, int NT, typename Epi, typename Epi2>
__global__ void __launch_bounds__(NT) k_gemm_pair(const __grid_constant__ CUtensorMap ta,
                                                  const __grid_constant__ CUtensorMap tb, GemmArgs g, Epi epi,
                                                  const __grid_constant__ CUtensorMap ta2,
                                                  const __grid_constant__ CUtensorMap tb2, GemmArgs g2, Epi2 epi2,
                                                  int tiles) {
    asm volatile("griddepcontrol.launch_dependents;");
    if ((int)blockIdx.x < tiles)
        gemm_tile<BN, NT>(ta, tb, g, blockIdx.x, epi);
    else
        gemm_tile<BN, NT>(ta2, tb2, g2, (int)blockIdx.x - tiles, epi2);
}

// ---- epilogues

__device__ __forceinline__ void store16(float* d, const float (&x)[16], bool aligned) {
    if (aligned) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            reinterpret_cast<float4*>(d)[i] = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = x[i];
    }
}

// 16 BF16 values of row `row` at column n, [rows x ld] row-major, and transposed [cols x ldT].
__device__ __forceinline__ void store16_bf16(__nv_bfloat16* d, __nv_bfloat16* dT, int row, int n, int ld, int ldT,
                                             const float (&x)[16]) {
    __align__(16) __nv_bfloat16 h[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) h[i] = __float2bfloat16_rn(x[i]);
    uint4* o = reinterpret_cast<uint4*>(d + (size_t)row * ld + n);  // ld and n are multiples of 16
    o[0] = reinterpret_cast<const uint4*>(h)[0];
    o[1] = reinterpret_cast<const uint4*>(h)[1];
    if (dT)
#pragma unroll
        for (int i = 0; i < 16; ++i) dT[(size_t)(n + i) * ldT + row] = h[i];  // a warp's rows: 64 bytes per column
}

// D = acc (+ bias), FP32.
struct EpiStore {
    static constexpr int THREADS = 128;
    float* D;
    int ldd;
    const float* bias;
    __device__ __forceinline__ void operator()(int row, int n, const uint32_t (&v)[16], bool live) const {
        if (!live) return;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]) + (bias ? bias[n + i] : 0.f);
        float* d = D + (size_t)row * ldd + n;
        store16(d, x, (reinterpret_cast<uintptr_t>(d) & 15) == 0);
    }
    __device__ __forceinline__ void finish(int) const {}
};

// cuTensorMapEncodeTiled from the driver, looked up once through the runtime.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// Tensor map of a row-major BF16 operand [rows x k] with leading dimension ld
// (elements): boxes of box_rows x 64, 128-byte swizzle, out-of-range elements
// read as zero.
static int operand_map(CUtensorMap* map, const __nv_bfloat16* base, int rows, int k, int ld, int box_rows) {
    auto enc = tensor_map_encoder();
    if (!enc) {
        set_error("mlp gemm: cuTensorMapEncodeTiled is not available from the driver");
        return TLFEA_CUDA_ERROR;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)GM_BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides,
                           box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("mlp gemm: tensor map encoding failed");
        return TLFEA_INVALID_ARG;
    }
    return TLFEA_OK;
}

// Column-tile width: the widest of 256 / 128 / 64 whose grid still covers the SMs
// (or 64 when even that does not).
static int gemm_tile_n(int M, int N, int sms) {
    const int mt = (M + MLP_TM - 1) / MLP_TM;
    for (int bn : {256, 128})
        if ((long long)mt * ((N + bn - 1) / bn) >= sms) return bn;
    return 64;
}

template <int BN, typename Epi>
static int gemm_launch_bn(const GemmArgs& g, const CUtensorMap& ta, const CUtensorMap& tb, const Epi& epi,
                          bool dependent, cudaStream_t st) {
    constexpr int NT = Epi::THREADS;
    auto kern = k_gemm_bf16<BN, NT, Epi>;
    // the shared-memory limit is a per-device attribute of the function: set it once per device
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    TLFEA_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        TLFEA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmGeom<BN>::SMEM));
        configured.fetch_or(bit);
    }
    const unsigned tiles = (unsigned)(((g.M + MLP_TM - 1) / MLP_TM) * ((g.N + BN - 1) / BN));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = GemmGeom<BN>::SMEM;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    TLFEA_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, g, epi));
    TLFEA_LAUNCHED(1);
    return TLFEA_OK;
}

template <int BN, typename Epi, typename Epi2>
static int gemm_launch_pair(const GemmArgs& g, const CUtensorMap& ta, const CUtensorMap& tb, const Epi& epi,
                            const GemmArgs& g2, const CUtensorMap& ta2, const CUtensorMap& tb2, const Epi2& epi2,
                            cudaStream_t st) {
    auto kern = k_gemm_pair<BN, 512, Epi, Epi2>;
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    TLFEA_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        TLFEA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmGeom<BN>::SMEM));
        configured.fetch_or(bit);
    }
    auto tiles = [](const GemmArgs& a) { return ((a.M + MLP_TM - 1) / MLP_TM) * ((a.N + BN - 1) / BN); };
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles(g) + tiles(g2)));
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = GemmGeom<BN>::SMEM;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TLFEA_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, g, epi, ta2, tb2, g2, epi2, tiles(g)));
    TLFEA_LAUNCHED(1);
    return TLFEA_OK;
}

// The device's SM count, asked once.
static int sm_count() {
    static std::atomic<int> sms{0};
    int n = sms.load();
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        sms.store(n);
    }
    return n;
}

// Launch with prepared operand maps (boxes of 128 and gemm_tile_n() rows).
template <typename Epi>
static int gemm_launch_maps(const GemmArgs& g, const CUtensorMap& ta, const CUtensorMap& tb, const Epi& epi,
                            bool dependent, cudaStream_t st) {
    const int bn = gemm_tile_n(g.M, g.N, sm_count());
    if (bn == 256) return gemm_launch_bn<256>(g, ta, tb, epi, dependent, st);
    if (bn == 128) return gemm_launch_bn<128>(g, ta, tb, epi, dependent, st);
    return gemm_launch_bn<64>(g, ta, tb, epi, dependent, st);
}

static int gemm_launch(const GemmArgs& g, cudaStream_t st) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.N % 16 || g.K % 16 || g.lda % 8 || g.ldb % 8 || g.lda < g.K ||
        g.ldb < g.K || (reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.B) & 15)) {
        set_error("mlp gemm: need N, K multiples of 16, leading dimensions >= K and multiples of 8, 16-byte "
                  "aligned operands");
        return TLFEA_INVALID_ARG;
    }
    CUtensorMap ta, tb;
    int s = operand_map(&ta, g.A, g.M, g.K, g.lda, MLP_TM);
    if (!s) s = operand_map(&tb, g.B, g.N, g.K, g.ldb, gemm_tile_n(g.M, g.N, sm_count()));
    if (s) return s;
    return gemm_launch_maps(g, ta, tb, EpiStore{g.D, g.ldd, g.bias}, false, st);
}

// ------------------------------------------------------------- elementwise

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// Input rows (FP32, din wide) -> BF16 [B x Kp] (zero padded) and its transpose [Kp x ldT].
__global__ void k_mlp_input(int B, int din, int Kp, const float* __restrict__ X, __nv_bfloat16* H,
                            __nv_bfloat16* HT, int ldT) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B * Kp) return;
    const int b = i / Kp, k = i - b * Kp;
    const __nv_bfloat16 v = __float2bfloat16_rn(k < din ? X[(size_t)b * din + k] : 0.f);
    H[i] = v;
    HT[(size_t)k * ldT + b] = v;
}

// ---- the network's epilogues.  Each was a launch of its own on the product's FP32 output (29
// launches a training step, bound by them); the arithmetic per element is the same.

// Z = acc + bias; H = GELU(Z) as BF16 in one or both layouts (the next layer's operands).
struct EpiAct {
    static constexpr int THREADS = 512;
    float* Z;
    int N;
    const float* bias;
    __nv_bfloat16* H;
    __nv_bfloat16* HT;
    int ldT;
    __device__ __forceinline__ void operator()(int row, int n, const uint32_t (&v)[16], bool live) const {
        if (!live) return;
        float z[16], h[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            z[i] = __uint_as_float(v[i]) + bias[n + i];
            h[i] = gelu(z[i]);
        }
        store16(Z + (size_t)row * N + n, z, true);
        store16_bf16(H, HT, row, n, N, ldT, h);
    }
    __device__ __forceinline__ void finish(int) const {}
};

// Sums of 16 values over the warp's 32 rows: lanes 2 j and 2 j + 1 end with the total of value j
// (halves exchanged, 16 shuffles).
__device__ __forceinline__ float warp_columns(float (&x)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = (lane & (2 * h)) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float give = up ? x[i] : x[i + h], keep = up ? x[i + h] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// Bias gradients start here: the column sums of dZ over 32 rows, cols[row / 32][N].
__device__ __forceinline__ void store_columns(float* cols, int N, int row, int n, const float (&d)[16]) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = d[i];
    const float s = warp_columns(x);
    const int lane = threadIdx.x & 31;
    if ((lane & 1) == 0) cols[(size_t)(row >> 5) * N + n + (lane >> 1)] = s;
}

// The output layer of a training step: Z, and of the mean squared error against T (M x N)
// dZ = 2 (Z - T) / (M N) as BF16 in both layouts, its column sums and the CTA's share of the loss.
struct EpiLoss {
    static constexpr int THREADS = 512;
    float* Z;
    int N;
    const float* bias;
    const float* T;
    float scale;  // 1 / (M N)
    __nv_bfloat16* dZ16;
    __nv_bfloat16* dZt16;
    int ldT;
    float* cols;
    float* part;  // per CTA
    float l;
    __device__ __forceinline__ void operator()(int row, int n, const uint32_t (&v)[16], bool live) {
        float d[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = 0.f;
        if (live) {
            float z[16];
            const size_t o = (size_t)row * N + n;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                z[i] = __uint_as_float(v[i]) + bias[n + i];
                const float e = z[i] - T[o + i];
                l += e * e * scale;
                d[i] = 2.0f * e * scale;
            }
            store16(Z + o, z, true);
            store16_bf16(dZ16, dZt16, row, n, N, ldT, d);
        }
        store_columns(cols, N, row, n, d);
    }
    __device__ __forceinline__ void finish(int tile) {
        __shared__ float red[32];
        const float s = block_sum(l, red);
        if (threadIdx.x == 0) part[tile] = s;
    }
};

// Input gradient: dZ = acc * GELU'(Z) of the layer below, BF16 in both layouts, and its column
// sums.
struct EpiGeluBack {
    static constexpr int THREADS = 512;
    const float* Z;
    int N;
    __nv_bfloat16* dZ16;
    __nv_bfloat16* dZt16;
    int ldT;
    float* cols;
    __device__ __forceinline__ void operator()(int row, int n, const uint32_t (&v)[16], bool live) const {
        float d[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = 0.f;
        if (live) {
            const float4* z4 = reinterpret_cast<const float4*>(Z + (size_t)row * N + n);
            float z[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 q = z4[i];
                z[4 * i] = q.x;
                z[4 * i + 1] = q.y;
                z[4 * i + 2] = q.z;
                z[4 * i + 3] = q.w;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] = __uint_as_float(v[i]) * gelu_grad(z[i]);
            store16_bf16(dZ16, dZt16, row, n, N, ldT, d);
        }
        store_columns(cols, N, row, n, d);
    }
    __device__ __forceinline__ void finish(int) const {}
};

// Weight gradient [Np x Kp].
struct EpiGrad {
    static constexpr int THREADS = 512;
    float* G;
    int Kp;
    __device__ __forceinline__ void operator()(int row, int n, const uint32_t (&v)[16], bool live) const {
        if (!live) return;
        float g[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) g[i] = __uint_as_float(v[i]);
        store16(G + (size_t)row * Kp + n, g, true);
    }
    __device__ __forceinline__ void finish(int) const {}
};

struct AdamWScalars {
    float lr, b1, b2, eps, wd, c1, c2;
};

// One AdamW update with bias-corrected moments.
__device__ __forceinline__ float adamw_update(float w, float g, float& m, float& v, const AdamWScalars& a, float wd) {
    m = a.b1 * m + (1.f - a.b1) * g;
    v = a.b2 * v + (1.f - a.b2) * g * g;
    return w - a.lr * (wd * w + (m / a.c1) / (sqrtf(v / a.c2) + a.eps));
}

// The end of a gradient or training step in one launch, up to MLP_END_LAYERS layers: bias
// gradients (the 32-row sums in order), the loss (the CTAs' shares in order) and, with STEP, the
// AdamW step of weights and biases and the weights' BF16 copies.  A layer's blocks: first its
// biases, 256 each, then its weights, 256 each.
constexpr int MLP_END_LAYERS = 8;
struct EndArgs {
    int layers, row_sums;            // row_sums: 32-row groups of the batch (whole tiles)
    int first[MLP_END_LAYERS + 1];   // first block of a layer
    int N[MLP_END_LAYERS], K[MLP_END_LAYERS], Kp[MLP_END_LAYERS];
    const float* cols[MLP_END_LAYERS];
    const float* gW[MLP_END_LAYERS];
    float *gb[MLP_END_LAYERS], *b[MLP_END_LAYERS], *mb[MLP_END_LAYERS], *vb[MLP_END_LAYERS];
    float *W[MLP_END_LAYERS], *mW[MLP_END_LAYERS], *vW[MLP_END_LAYERS];
    __nv_bfloat16 *W16[MLP_END_LAYERS], *Wt16[MLP_END_LAYERS];
    const float* loss_part;
    int loss_n;
    float* loss;
    AdamWScalars a;
};
template <bool STEP>
__global__ void __launch_bounds__(256) k_mlp_end(EndArgs A) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int l = 0;
    while (l + 1 < A.layers && (int)blockIdx.x >= A.first[l + 1]) ++l;
    const int N = A.N[l], bias_blocks = (N + 255) / 256, blk = (int)blockIdx.x - A.first[l];
    if (blk < bias_blocks) {
        const int n = blk * 256 + threadIdx.x;
        if (n < N) {
            float t = 0.f;
#pragma unroll 8
            for (int k = 0; k < A.row_sums; ++k) t += A.cols[l][(size_t)k * N + n];
            A.gb[l][n] = t;
            if constexpr (STEP) {
                float m = A.mb[l][n], v = A.vb[l][n];
                A.b[l][n] = adamw_update(A.b[l][n], t, m, v, A.a, 0.f);
                A.mb[l][n] = m;
                A.vb[l][n] = v;
            }
        }
        if (blockIdx.x == 0 && threadIdx.x < 32 && A.loss) {
            float t = 0.f;
            for (int k = threadIdx.x; k < A.loss_n; k += 32) t += A.loss_part[k];
            t = warp_sum(t);
            if (threadIdx.x == 0) *A.loss = t;
        }
        return;
    }
    if constexpr (STEP) {
        const int Kp = A.Kp[l], i = (blk - bias_blocks) * 256 + threadIdx.x;
        if (i >= N * Kp) return;
        const int n = i / Kp, k = i - n * Kp;
        if (k >= A.K[l]) return;  // padding stays zero
        float m = A.mW[l][i], v = A.vW[l][i];
        const float w = adamw_update(A.W[l][i], A.gW[l][i], m, v, A.a, A.a.wd);
        A.mW[l][i] = m;
        A.vW[l][i] = v;
        A.W[l][i] = w;
        const __nv_bfloat16 h = __float2bfloat16_rn(w);
        A.W16[l][i] = h;
        A.Wt16[l][(size_t)k * N + n] = h;
    }
}

// AdamW on an [N x Kreal] weight (stored with Kp columns) or a bias (Kp = 0); refreshes the
// BF16 copies W [N x Kp] and W^T [Kp x N].
__global__ void k_mlp_adamw(int N, int Kreal, int Kp, float* W, const float* __restrict__ G, int ldg, float* m,
                            float* v, __nv_bfloat16* W16, __nv_bfloat16* Wt16, AdamWScalars a, float wd) {
    const int cols = Kp > 0 ? Kp : 1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N * cols) return;
    const int n = i / cols, k = i - n * cols;
    if (Kp > 0 && k >= Kreal) return;  // padding stays zero
    const float g = G[(size_t)n * ldg + k];
    float mi = m[i], vi = v[i];
    const float w = adamw_update(W[i], g, mi, vi, a, wd);
    m[i] = mi;
    v[i] = vi;
    W[i] = w;
    if (W16) {
        const __nv_bfloat16 h = __float2bfloat16_rn(w);
        W16[i] = h;
        Wt16[(size_t)k * N + n] = h;
    }
}

__global__ void k_mlp_to_bf16(int N, int Kp, const float* __restrict__ W, __nv_bfloat16* W16, __nv_bfloat16* Wt16) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N * Kp) return;
    const int n = i / Kp, k = i - n * Kp;
    const __nv_bfloat16 h = __float2bfloat16_rn(W[i]);
    W16[i] = h;
    Wt16[(size_t)k * N + n] = h;
}

}  // namespace tlfea

using namespace tlfea;

struct tlfea_mlp_s {
    int L = 0;
    std::vector<int> dims, Kp, Np;  // Kp: padded input width, Np: output rows padded to 128
    int Bmax = 0;
    int device = 0;
    cudaStream_t stream = nullptr;
    int* err = nullptr;
    std::vector<float*> W, b, mW, vW, mb, vb, gW, gb, Z;
    std::vector<__nv_bfloat16*> W16, Wt16, H, HT;  // H[l], HT[l]: input of layer l
    std::vector<__nv_bfloat16*> dZ16, dZt16;  // per layer: output gradients, both layouts
    std::vector<float*> cols;                 // and their column sums over 32 rows each
    float *part = nullptr, *loss = nullptr, *xin = nullptr, *tin = nullptr;
    // operand maps of the products at batch size map_batch: forward, input gradient, weight gradient
    struct Maps {
        CUtensorMap a, b;
    };
    std::vector<Maps> fwd, gx, gw;
    int map_batch = 0;
    int maxN = 0;
    long long step = 0;
    bool grads_valid = false;
};

namespace {

int mlp_check_err(tlfea_mlp_s* m) {
    int e = 0;
    TLFEA_CUDA(cudaMemcpyAsync(&e, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    TLFEA_CUDA(cudaStreamSynchronize(m->stream));
    if (e) {
        cudaMemsetAsync(m->err, 0, sizeof(int), m->stream);
        set_error("mlp: a tensor-core product did not complete (bounded wait ran out)");
        return TLFEA_CUDA_ERROR;
    }
    return TLFEA_OK;
}

inline unsigned grid1(long long n, int bs = 256) { return (unsigned)((n + bs - 1) / bs); }

GemmArgs fwd_args(const tlfea_mlp_s* m, int l, int B) {
    return GemmArgs{B, m->dims[l + 1], m->Kp[l], m->H[l], m->Kp[l], m->W16[l], m->Kp[l], nullptr, nullptr, 0, m->err};
}
// dH [B x Kp] = dZ x W (= dZ x (W^T)^T)
GemmArgs gx_args(const tlfea_mlp_s* m, int l, int B) {
    const int N = m->dims[l + 1];
    return GemmArgs{B, m->Kp[l], N, m->dZ16[l], N, m->Wt16[l], N, nullptr, nullptr, 0, m->err};
}
// gW [Np x Kp] = dZ^T (rows padded with zeros) x H
GemmArgs gw_args(const tlfea_mlp_s* m, int l, int B) {
    return GemmArgs{m->Np[l], m->Kp[l], B, m->dZt16[l], m->Bmax, m->HT[l], m->Bmax, nullptr, nullptr, 0, m->err};
}

// The operand maps at this batch size (encoded once, not per product and call).
int mlp_maps(tlfea_mlp_s* m, int B) {
    if (m->map_batch == B) return TLFEA_OK;
    m->map_batch = 0;
    m->fwd.resize(m->L);
    m->gx.resize(m->L);
    m->gw.resize(m->L);
    auto encode = [](tlfea_mlp_s::Maps& k, const GemmArgs& g) -> int {
        int s = operand_map(&k.a, g.A, g.M, g.K, g.lda, MLP_TM);
        if (!s) s = operand_map(&k.b, g.B, g.N, g.K, g.ldb, gemm_tile_n(g.M, g.N, sm_count()));
        return s;
    };
    for (int l = 0; l < m->L; ++l) {
        int s = encode(m->fwd[l], fwd_args(m, l, B));
        if (!s && B % 16 == 0) s = encode(m->gw[l], gw_args(m, l, B));  // a training batch
        if (!s && l > 0) s = encode(m->gx[l], gx_args(m, l, B));
        if (s) return s;
    }
    m->map_batch = B;
    return TLFEA_OK;
}

// Activations of a batch; with T (a training step) the output layer's epilogue forms the loss
// and its gradient too.
int mlp_forward(tlfea_mlp_s* m, const float* X, int B, const float* T) {
    cudaStream_t st = m->stream;
    int s = mlp_maps(m, B);
    if (s) return s;
    k_mlp_input<<<grid1((long long)B * m->Kp[0]), 256, 0, st>>>(B, m->dims[0], m->Kp[0], X, m->H[0], m->HT[0], m->Bmax);
    TLFEA_CHECK_LAUNCH();
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1];
        const GemmArgs g = fwd_args(m, l, B);
        if (l + 1 < m->L)
            s = gemm_launch_maps(g, m->fwd[l].a, m->fwd[l].b,
                                 EpiAct{m->Z[l], N, m->b[l], m->H[l + 1], T ? m->HT[l + 1] : nullptr, m->Bmax}, true, st);
        else if (T)
            s = gemm_launch_maps(g, m->fwd[l].a, m->fwd[l].b,
                                 EpiLoss{m->Z[l], N, m->b[l], T, 1.0f / ((float)B * (float)N), m->dZ16[l], m->dZt16[l],
                                         m->Bmax, m->cols[l], m->part, 0.f},
                                 true, st);
        else
            s = gemm_launch_maps(g, m->fwd[l].a, m->fwd[l].b, EpiStore{m->Z[l], N, m->b[l]}, true, st);
        if (s) return s;
    }
    return TLFEA_OK;
}

// Gradients of the batch whose activations and output gradient stand; with a, the AdamW step.
int mlp_backward(tlfea_mlp_s* m, int B, const AdamWScalars* a) {
    cudaStream_t st = m->stream;
    const int L = m->L;
    for (int l = L - 1; l >= 0; --l) {
        const GemmArgs gw = gw_args(m, l, B);
        const EpiGrad grad{m->gW[l], m->Kp[l]};
        int s = TLFEA_OK;
        if (l > 0) {
            const GemmArgs gx = gx_args(m, l, B);
            const EpiGeluBack back{m->Z[l - 1], m->dims[l], m->dZ16[l - 1], m->dZt16[l - 1], m->Bmax, m->cols[l - 1]};
            if (gemm_tile_n(gx.M, gx.N, sm_count()) == 64 && gemm_tile_n(gw.M, gw.N, sm_count()) == 64) {
                s = gemm_launch_pair<64>(gx, m->gx[l].a, m->gx[l].b, back, gw, m->gw[l].a, m->gw[l].b, grad, st);
                if (s) return s;
                continue;
            }
            s = gemm_launch_maps(gx, m->gx[l].a, m->gx[l].b, back, true, st);
        }
        if (!s) s = gemm_launch_maps(gw, m->gw[l].a, m->gw[l].b, grad, true, st);
        if (s) return s;
    }
    const int Nout = m->dims[L], bn = gemm_tile_n(B, Nout, sm_count()), row_tiles = (B + MLP_TM - 1) / MLP_TM;
    for (int l0 = 0; l0 < L; l0 += MLP_END_LAYERS) {
        EndArgs A{};
        A.layers = std::min(MLP_END_LAYERS, L - l0);
        A.row_sums = row_tiles * (MLP_TM / 32);
        for (int k = 0; k < A.layers; ++k) {
            const int l = l0 + k, N = m->dims[l + 1];
            A.first[k + 1] = A.first[k] + (N + 255) / 256 + (a ? (N * m->Kp[l] + 255) / 256 : 0);
            A.N[k] = N;
            A.K[k] = m->dims[l];
            A.Kp[k] = m->Kp[l];
            A.cols[k] = m->cols[l];
            A.gW[k] = m->gW[l];
            A.gb[k] = m->gb[l];
            A.b[k] = m->b[l];
            A.mb[k] = m->mb[l];
            A.vb[k] = m->vb[l];
            A.W[k] = m->W[l];
            A.mW[k] = m->mW[l];
            A.vW[k] = m->vW[l];
            A.W16[k] = m->W16[l];
            A.Wt16[k] = m->Wt16[l];
        }
        A.loss_part = m->part;
        A.loss_n = row_tiles * ((Nout + bn - 1) / bn);
        A.loss = l0 == 0 ? m->loss : nullptr;
        if (a) A.a = *a;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)A.first[A.layers]);
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        TLFEA_CUDA(a ? cudaLaunchKernelEx(&cfg, k_mlp_end<true>, A) : cudaLaunchKernelEx(&cfg, k_mlp_end<false>, A));
        TLFEA_LAUNCHED(1);
    }
    return TLFEA_OK;
}

AdamWScalars next_step(tlfea_mlp_s* m, float lr, float b1, float b2, float eps, float wd) {
    m->step += 1;
    return AdamWScalars{lr, b1, b2, eps, wd, 1.0f - powf(b1, (float)m->step), 1.0f - powf(b2, (float)m->step)};
}

int mlp_adamw(tlfea_mlp_s* m, float lr, float b1, float b2, float eps, float wd) {
    cudaStream_t st = m->stream;
    const AdamWScalars a = next_step(m, lr, b1, b2, eps, wd);
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1], K = m->dims[l], Kp = m->Kp[l];
        k_mlp_adamw<<<grid1((long long)N * Kp), 256, 0, st>>>(N, K, Kp, m->W[l], m->gW[l], Kp, m->mW[l], m->vW[l],
                                                              m->W16[l], m->Wt16[l], a, wd);
        TLFEA_CHECK_LAUNCH();
        k_mlp_adamw<<<grid1(N), 256, 0, st>>>(N, 1, 0, m->b[l], m->gb[l], 1, m->mb[l], m->vb[l], nullptr, nullptr, a,
                                              0.f);
        TLFEA_CHECK_LAUNCH();
    }
    return TLFEA_OK;
}

int mlp_refresh_bf16(tlfea_mlp_s* m) {
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1], Kp = m->Kp[l];
        k_mlp_to_bf16<<<grid1((long long)N * Kp), 256, 0, m->stream>>>(N, Kp, m->W[l], m->W16[l], m->Wt16[l]);
        TLFEA_CHECK_LAUNCH();
    }
    return TLFEA_OK;
}

long long mlp_param_count(const tlfea_mlp_s* m) {
    long long n = 0;
    for (int l = 0; l < m->L; ++l) n += (long long)m->dims[l + 1] * m->dims[l] + m->dims[l + 1];
    return n;
}

}  // namespace

#define CHECK_MLP(m)                  \
    do {                              \
        if (!(m)) {                   \
            set_error("null mlp");    \
            return TLFEA_INVALID_ARG; \
        }                             \
    } while (0)

extern "C" {

int tlfea_mlp_gemm_bf16(int M, int N, int K, const void* d_a, int lda, const void* d_b, int ldb, const float* d_bias,
                        float* d_d, int ldd, void* stream) {
    int* err = nullptr;
    int s = dalloc(&err, 1);
    if (s) return s;
    cudaStream_t st = (cudaStream_t)stream;
    TLFEA_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    GemmArgs g{M, N, K, (const __nv_bfloat16*)d_a, lda, (const __nv_bfloat16*)d_b, ldb, d_bias, d_d, ldd, err};
    s = gemm_launch(g, st);
    int e = 0;
    if (!s && cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
        cudaStreamSynchronize(st) == cudaSuccess && e) {
        set_error("mlp gemm: bounded wait ran out");
        s = TLFEA_CUDA_ERROR;
    }
    cudaStreamSynchronize(st);
    dfree(err);
    return s;
}

int tlfea_mlp_gemm_bf16_async(int M, int N, int K, const void* d_a, int lda, const void* d_b, int ldb,
                              const float* d_bias, float* d_d, int ldd, int* d_err, void* stream) {
    if (!d_err || !d_d) {
        set_error("mlp gemm: null output or error flag");
        return TLFEA_INVALID_ARG;
    }
    GemmArgs g{M, N, K, (const __nv_bfloat16*)d_a, lda, (const __nv_bfloat16*)d_b, ldb, d_bias, d_d, ldd, d_err};
    return gemm_launch(g, (cudaStream_t)stream);
}

int tlfea_mlp_create(int n_layers, const int* dims, int max_batch, unsigned long long seed, tlfea_mlp* out) {
    if (!out || !dims || n_layers < 1 || max_batch <= 0 || max_batch % 128) {
        set_error("mlp_create: need >= 1 layer and max_batch a positive multiple of 128");
        return TLFEA_INVALID_ARG;
    }
    for (int l = 1; l <= n_layers; ++l)
        if (dims[l] <= 0 || dims[l] % 16 || dims[l] > 4096) {
            set_error("mlp_create: layer widths must be positive multiples of 16 (<= 4096)");
            return TLFEA_INVALID_ARG;
        }
    if (dims[0] <= 0 || dims[0] > 4096) return TLFEA_INVALID_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device");
        return TLFEA_NO_CUDA_DEVICE;
    }
    tlfea_mlp_s* m = new tlfea_mlp_s();
    cudaGetDevice(&m->device);
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete m;
        set_error("cudaStreamCreate failed");
        return TLFEA_CUDA_ERROR;
    }
    m->L = n_layers;
    m->dims.assign(dims, dims + n_layers + 1);
    m->Bmax = max_batch;
    for (int l = 0; l < n_layers; ++l) {
        m->Kp.push_back((dims[l] + 15) / 16 * 16);
        m->Np.push_back((dims[l + 1] + MLP_TM - 1) / MLP_TM * MLP_TM);
        m->maxN = std::max(m->maxN, dims[l + 1]);
    }
    const int L = n_layers, B = max_batch;
    m->W.assign(L, nullptr); m->b.assign(L, nullptr); m->mW.assign(L, nullptr); m->vW.assign(L, nullptr);
    m->mb.assign(L, nullptr); m->vb.assign(L, nullptr); m->gW.assign(L, nullptr); m->gb.assign(L, nullptr);
    m->Z.assign(L, nullptr); m->W16.assign(L, nullptr); m->Wt16.assign(L, nullptr);
    m->H.assign(L, nullptr); m->HT.assign(L, nullptr);
    m->cols.assign(L, nullptr); m->dZ16.assign(L, nullptr); m->dZt16.assign(L, nullptr);
    int s = dalloc(&m->err, 1);
    for (int l = 0; l < L && !s; ++l) {
        const size_t nk = (size_t)dims[l + 1] * m->Kp[l];
        s = dalloc(&m->W[l], nk) | dalloc(&m->mW[l], nk) | dalloc(&m->vW[l], nk) |
            dalloc(&m->gW[l], (size_t)m->Np[l] * m->Kp[l]) | dalloc(&m->b[l], dims[l + 1]) |
            dalloc(&m->mb[l], dims[l + 1]) | dalloc(&m->vb[l], dims[l + 1]) | dalloc(&m->gb[l], dims[l + 1]) |
            dalloc(&m->Z[l], (size_t)B * dims[l + 1]) | dalloc(&m->W16[l], nk) | dalloc(&m->Wt16[l], nk) |
            dalloc(&m->H[l], (size_t)B * m->Kp[l]) | dalloc(&m->HT[l], (size_t)m->Kp[l] * B) |
            dalloc(&m->dZ16[l], (size_t)B * dims[l + 1]) | dalloc(&m->dZt16[l], (size_t)m->Np[l] * B) |
            dalloc(&m->cols[l], (size_t)(B / 32) * dims[l + 1]);
    }
    if (!s)
        s = dalloc(&m->part, (size_t)(B * m->maxN + 255) / 256 + 1) | dalloc(&m->loss, 1) |
            dalloc(&m->xin, (size_t)B * dims[0]) | dalloc(&m->tin, (size_t)B * dims[L]);
    if (s) {
        tlfea_mlp_destroy(m);
        return TLFEA_CUDA_ERROR;
    }
    // zero everything the padding relies on (padded weight columns, padded
    // gradient rows), then a seeded uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) init
    cudaStream_t st = m->stream;
    cudaMemsetAsync(m->err, 0, sizeof(int), st);
    for (int l = 0; l < L; ++l) {
        cudaMemsetAsync(m->dZt16[l], 0, (size_t)m->Np[l] * B * sizeof(__nv_bfloat16), st);
        const size_t nk = (size_t)dims[l + 1] * m->Kp[l];
        cudaMemsetAsync(m->mW[l], 0, nk * 4, st);
        cudaMemsetAsync(m->vW[l], 0, nk * 4, st);
        cudaMemsetAsync(m->mb[l], 0, dims[l + 1] * 4, st);
        cudaMemsetAsync(m->vb[l], 0, dims[l + 1] * 4, st);
        cudaMemsetAsync(m->H[l], 0, (size_t)B * m->Kp[l] * 2, st);
        cudaMemsetAsync(m->HT[l], 0, (size_t)m->Kp[l] * B * 2, st);
    }
    std::vector<float> flat((size_t)mlp_param_count(m));
    unsigned long long x = seed * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
    auto next = [&]() {  // splitmix64
        x += 0x9E3779B97F4A7C15ull;
        unsigned long long z = x;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    size_t o = 0;
    for (int l = 0; l < L; ++l) {
        const float bound = 1.0f / std::sqrt((float)dims[l]);
        const size_t cnt = (size_t)dims[l + 1] * dims[l] + dims[l + 1];
        for (size_t i = 0; i < cnt; ++i) flat[o + i] = bound * (2.0f * (float)((next() >> 11) * 0x1.0p-53) - 1.0f);
        o += cnt;
    }
    cudaStreamSynchronize(st);
    s = tlfea_mlp_set_params(m, flat.data(), (long long)flat.size());
    if (s) {
        tlfea_mlp_destroy(m);
        return s;
    }
    *out = m;
    return TLFEA_OK;
}

int tlfea_mlp_destroy(tlfea_mlp m) {
    CHECK_MLP(m);
    TLFEA_CUDA(cudaSetDevice(m->device));
    if (m->stream) cudaStreamSynchronize(m->stream);
    for (auto* v : {&m->W, &m->b, &m->mW, &m->vW, &m->mb, &m->vb, &m->gW, &m->gb, &m->Z, &m->cols})
        for (auto& p : *v) dfree(p);
    for (auto* v : {&m->W16, &m->Wt16, &m->H, &m->HT, &m->dZ16, &m->dZt16})
        for (auto& p : *v) dfree(p);
    dfree(m->part); dfree(m->loss); dfree(m->xin); dfree(m->tin);
    dfree(m->err);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return TLFEA_OK;
}

int tlfea_mlp_get_stream(tlfea_mlp m, void** stream) {
    CHECK_MLP(m);
    if (!stream) return TLFEA_INVALID_ARG;
    *stream = (void*)m->stream;
    return TLFEA_OK;
}

int tlfea_mlp_param_count(tlfea_mlp m, long long* n) {
    CHECK_MLP(m);
    if (!n) return TLFEA_INVALID_ARG;
    *n = mlp_param_count(m);
    return TLFEA_OK;
}

// Flat FP32 parameters: per layer W [dims[l+1] x dims[l]] row-major, then b.
int tlfea_mlp_set_params(tlfea_mlp m, const float* p, long long n) {
    CHECK_MLP(m);
    if (!p || n != mlp_param_count(m)) {
        set_error("mlp_set_params: size mismatch");
        return TLFEA_SIZE_MISMATCH;
    }
    size_t o = 0;
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1], K = m->dims[l], Kp = m->Kp[l];
        std::vector<float> w((size_t)N * Kp, 0.f);
        for (int r = 0; r < N; ++r)
            for (int k = 0; k < K; ++k) w[(size_t)r * Kp + k] = p[o + (size_t)r * K + k];
        o += (size_t)N * K;
        TLFEA_CUDA(cudaMemcpyAsync(m->W[l], w.data(), w.size() * 4, cudaMemcpyHostToDevice, m->stream));
        TLFEA_CUDA(cudaMemcpyAsync(m->b[l], p + o, (size_t)N * 4, cudaMemcpyHostToDevice, m->stream));
        o += N;
        TLFEA_CUDA(cudaStreamSynchronize(m->stream));
    }
    const int s = mlp_refresh_bf16(m);
    if (s) return s;
    TLFEA_CUDA(cudaStreamSynchronize(m->stream));
    return TLFEA_OK;
}

int tlfea_mlp_get_params(tlfea_mlp m, float* p, long long n) {
    CHECK_MLP(m);
    if (!p || n != mlp_param_count(m)) {
        set_error("mlp_get_params: size mismatch");
        return TLFEA_SIZE_MISMATCH;
    }
    size_t o = 0;
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1], K = m->dims[l], Kp = m->Kp[l];
        std::vector<float> w((size_t)N * Kp);
        TLFEA_CUDA(cudaMemcpyAsync(w.data(), m->W[l], w.size() * 4, cudaMemcpyDeviceToHost, m->stream));
        TLFEA_CUDA(cudaMemcpyAsync(p + o + (size_t)N * K, m->b[l], (size_t)N * 4, cudaMemcpyDeviceToHost, m->stream));
        TLFEA_CUDA(cudaStreamSynchronize(m->stream));
        for (int r = 0; r < N; ++r)
            for (int k = 0; k < K; ++k) p[o + (size_t)r * K + k] = w[(size_t)r * Kp + k];
        o += (size_t)N * K + N;
    }
    return TLFEA_OK;
}

// Gradients of the last loss_grad call, in the parameter layout.
int tlfea_mlp_get_grads(tlfea_mlp m, float* g, long long n) {
    CHECK_MLP(m);
    if (!g || n != mlp_param_count(m)) {
        set_error("mlp_get_grads: size mismatch");
        return TLFEA_SIZE_MISMATCH;
    }
    if (!m->grads_valid) {
        set_error("mlp_get_grads: no gradients computed yet");
        return TLFEA_NOT_SETUP;
    }
    size_t o = 0;
    for (int l = 0; l < m->L; ++l) {
        const int N = m->dims[l + 1], K = m->dims[l], Kp = m->Kp[l];
        std::vector<float> w((size_t)m->Np[l] * Kp);
        TLFEA_CUDA(cudaMemcpyAsync(w.data(), m->gW[l], w.size() * 4, cudaMemcpyDeviceToHost, m->stream));
        TLFEA_CUDA(cudaMemcpyAsync(g + o + (size_t)N * K, m->gb[l], (size_t)N * 4, cudaMemcpyDeviceToHost, m->stream));
        TLFEA_CUDA(cudaStreamSynchronize(m->stream));
        for (int r = 0; r < N; ++r)
            for (int k = 0; k < K; ++k) g[o + (size_t)r * K + k] = w[(size_t)r * Kp + k];
        o += (size_t)N * K + N;
    }
    return TLFEA_OK;
}

// y[batch x dims[L]] = MLP(x[batch x dims[0]]), device pointers, on the MLP stream.
int tlfea_mlp_forward(tlfea_mlp m, const float* d_x, int batch, float* d_y) {
    CHECK_MLP(m);
    if (!d_x || !d_y || batch <= 0 || batch > m->Bmax) return TLFEA_INVALID_ARG;
    int s = mlp_forward(m, d_x, batch, nullptr);
    if (s) return s;
    const int Nout = m->dims[m->L];
    TLFEA_CUDA(cudaMemcpyAsync(d_y, m->Z[m->L - 1], (size_t)batch * Nout * 4, cudaMemcpyDeviceToDevice, m->stream));
    return mlp_check_err(m);
}

// Forward + backward of the mean squared error against d_t; keeps the
// gradients; *loss (host) = the batch loss.  batch must be a multiple of 16.
int tlfea_mlp_loss_grad(tlfea_mlp m, const float* d_x, const float* d_t, int batch, float* loss) {
    CHECK_MLP(m);
    if (!d_x || !d_t || batch <= 0 || batch > m->Bmax || batch % 16) {
        set_error("mlp_loss_grad: batch must be a positive multiple of 16 up to max_batch");
        return TLFEA_INVALID_ARG;
    }
    int s = mlp_forward(m, d_x, batch, d_t);
    if (!s) s = mlp_backward(m, batch, nullptr);
    if (s) return s;
    if (loss) TLFEA_CUDA(cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->stream));
    s = mlp_check_err(m);
    if (s) return s;
    m->grads_valid = true;
    return TLFEA_OK;
}

int tlfea_mlp_adamw_step(tlfea_mlp m, float lr, float beta1, float beta2, float eps, float weight_decay) {
    CHECK_MLP(m);
    if (!m->grads_valid) {
        set_error("mlp_adamw_step: no gradients computed yet");
        return TLFEA_NOT_SETUP;
    }
    const int s = mlp_adamw(m, lr, beta1, beta2, eps, weight_decay);
    if (s) return s;
    return TLFEA_OK;
}

// One optimisation step on a minibatch: forward, backward, AdamW.  With
// loss == NULL nothing is read back (no host synchronisation).
int tlfea_mlp_train_step(tlfea_mlp m, const float* d_x, const float* d_t, int batch, float lr, float beta1,
                         float beta2, float eps, float weight_decay, float* loss) {
    CHECK_MLP(m);
    if (!d_x || !d_t || batch <= 0 || batch > m->Bmax || batch % 16) {
        set_error("mlp_train_step: batch must be a positive multiple of 16 up to max_batch");
        return TLFEA_INVALID_ARG;
    }
    int s = mlp_forward(m, d_x, batch, d_t);
    if (!s) {
        const AdamWScalars a = next_step(m, lr, beta1, beta2, eps, weight_decay);
        s = mlp_backward(m, batch, &a);
    }
    if (s) return s;
    m->grads_valid = true;
    if (loss) {
        TLFEA_CUDA(cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->stream));
        return mlp_check_err(m);
    }
    return TLFEA_OK;
}

int tlfea_mlp_sync(tlfea_mlp m) {
    CHECK_MLP(m);
    return mlp_check_err(m);
}

}  // extern "C"

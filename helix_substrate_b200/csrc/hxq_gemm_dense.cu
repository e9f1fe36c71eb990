// hxq_gemm, many tokens: the second of two passes.  hxq_gemm.cu first writes a run of weight rows as
// bf16 (codebook, affine and sidecar applied in fp32, rounded once: the operand the fused kernels
// build tile by tile) into scratch, then this kernel multiplies
//
//   y[m, o] = sum_k x[m, k] * W[o, k] + bias[o]        (bf16 operands, fp32 accumulator in TMEM)
//
// Bound by the tensor cores, four fifths of the time, and by the staging of their operands (measured below).  A pair
// of CTAs (one TPC) owns a 256-token x BN-row tile, cta_group::2:
//
//   * the weight rows come blocked, [K / 64][rows][64]: a stage's box is one contiguous piece (as 128-byte
//     rows 2 K bytes apart a box took several microseconds from HBM, and a product with few token
//     tiles, which streams the weights rather than re-reads them, ran at that latency);
//   * each CTA stages its own 128 tokens and its own half of the BN weight rows (TMA, 128-byte
//     swizzle, 64 columns a stage) and reports to the leader's barrier, so a stage costs one SM
//     16 KB + BN * 64 bytes of shared memory traffic instead of the 16 KB + BN * 128 of a lone CTA:
//     at BN = 256 a lone CTA's copies and operand reads are above what shared memory moves in the
//     time of the MMAs, the pair's are not;
//   * the leader's MMA lane issues four tcgen05.mma (M = 256, N = BN, K = 16) per stage; the commit
//     frees the stage in both CTAs;
//   * the accumulator is double-buffered (2 x 256 columns): four warps per CTA drain one tile while
//     the next one is multiplied;
//   * persistent: one pair per TPC walks the tiles in groups of eight token tiles, so that the
//     tiles running at one time share operands in L2.
//
// Measured: 1.46 PFLOP/s on [18944 x 3584] at 2048 and 8192 tokens.  A 64-column step of a pair's 256 x 256 tile takes
// 673 cycles (0.43 us at the 1.6 GHz of that load), the tensor pipe being active for 550 of them; in the rest the
// next stage is waited for, 32 KB per SM and step, 11 TB/s over the GPU.  (The library's product reaches 1.64 PFLOP/s.)
//
// BN is a launch argument, a multiple of 32 up to 256 (see pick_tile): an output width that leaves a
// nearly empty last wave at 256 columns takes the width that fills it.
// Every mbarrier wait is bounded and raises the status word.  No multicast loads.

#include <cuda.h>

#include "hxq_common.cuh"
#include "hxq_sm100.cuh"

namespace hxq {
namespace gemm {
bool make_map_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t outer,
                 uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw);
}  // namespace gemm

namespace gemmd {

constexpr int TM = 256;                    // tokens per pair
constexpr int BK = 64;                     // K per stage: one 128-byte swizzled row
constexpr int BN_MAX = 256;
constexpr int MAX_STAGES = 11;
constexpr int A_BYTES = (TM / 2) * BK * 2;           // 16 KB: this CTA's 128 tokens
constexpr int RING_BYTES = 220 * 1024;               // as many stages of A_BYTES + BN * 64 as fit
constexpr int SMEM_TOTAL = RING_BYTES + 256 + 1024;  // barriers, slack for 1024-byte alignment
constexpr int stages_for(int bn) { return RING_BYTES / (A_BYTES + bn * BK) < MAX_STAGES ? RING_BYTES / (A_BYTES + bn * BK) : MAX_STAGES; }
constexpr int EPI_WARPS = 4;
constexpr int NUM_THREADS = 32 * (2 + EPI_WARPS);
constexpr int TMEM_COLS = 512;
constexpr int GROUP_M = 8;                 // token tiles walked together

struct Args {
    const float* bias;      // of the first row of this run, or nullptr
    void* y;                // column of the first row of this run
    int32_t* status;
    int64_t ldy;
    int32_t M, N, k_steps;  // tokens, weight rows of this run, 64-column steps
    int32_t tiles_m, tiles_n, bn, stages;
    int32_t y_dtype, vec;   // vec: rows of y can take 16-byte stores
};

__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A stage's copy into this CTA's shared memory, reporting to a barrier that may be the other CTA's.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One arrival on this barrier of both CTAs when the MMAs issued so far have retired.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(sm100::smem_u32(bar)), "h"((uint16_t)3)
        : "memory");
}

// As sm100::mbar_wait, for arrivals that come from the other CTA.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort) {
    const long long t0 = clock64();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(sm100::smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort != 0) return false;
        if (clock64() - t0 > 2000000000LL) {
            *abort = 1;
            return false;
        }
    }
}

// Tile number -> (token tile, row tile): groups of GROUP_M token tiles, token tile fastest inside.
__device__ __forceinline__ void tile_at(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
    const int per_group = GROUP_M * tiles_n;
    const int g = t / per_group, rem = t - g * per_group;
    const int first = g * GROUP_M;
    const int size = tiles_m - first < GROUP_M ? tiles_m - first : GROUP_M;
    tn = rem / size;
    tm = first + rem - tn * size;
}

__device__ __forceinline__ uint32_t pack16(float lo, float hi, int dt) {
    if (dt == HXQ_BF16) {
        __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_dense_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Args a) {
    extern __shared__ char smem_raw[];
    char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + RING_BYTES);   // [stages] both CTAs' copies landed (the leader's is used)
    uint64_t* empty = full + MAX_STAGES;        // [stages] MMAs of the stage retired
    uint64_t* acc_full = empty + MAX_STAGES;    // [2] accumulator complete
    uint64_t* acc_empty = acc_full + 2;     // [2] accumulator read by both CTAs (the leader's is used)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= 256, "barrier area");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cta_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles = a.tiles_m * a.tiles_n;
    const int bn = a.bn, stages = a.stages;
    const int stage_bytes = A_BYTES + bn * BK;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            sm100::mbar_init(&full[s], 1);
            sm100::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            sm100::mbar_init(&acc_full[b], 1);
            sm100::mbar_init(&acc_empty[b], 2 * EPI_WARPS);
        }
        *abort_flag = 0;
        sm100::fence_barrier_init();
        sm100::prefetch_tensormap(&map_x);
        sm100::prefetch_tensormap(&map_w);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm100::smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    cluster_sync();       // the other CTA's barriers and tensor memory are ready too
    sm100::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");     // the weight rows are written

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (each CTA its own operands)
        if (lane == 0) {
            const uint32_t tx = 2u * (uint32_t)(A_BYTES + bn * BK);     // both CTAs' bytes of a stage
            int s = 0;
            uint32_t ph = 0;        // stage, and the parity of its round
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs) {
                int tm, tn;
                tile_at(t, a.tiles_m, a.tiles_n, tm, tn);
                const int ym = tm * TM + (int)rank * (TM / 2), yn = tn * bn + (int)rank * (bn / 2);
                for (int ks = 0; ks < a.k_steps; ++ks) {
                    ok = sm100::mbar_wait(&empty[s], ph ^ 1u, abort_flag);
                    if (!ok) break;
                    if (rank == 0) sm100::mbar_arrive_expect_tx(&full[s], tx);
                    const uint32_t bar = map_to_rank(sm100::smem_u32(&full[s]), 0);
                    const uint32_t st = sm100::smem_u32(smem + s * stage_bytes);
                    tma_load_2d_pair(st, &map_x, bar, ks * BK, ym);
                    tma_load_2d_pair(st + A_BYTES, &map_w, bar, 0, ks * a.N + yn);
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ok) {     // gave up: let copies already in flight land before the pair retires
                const long long t0 = clock64();
                while (clock64() - t0 < 20000000LL) { }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader)
        if (rank == 0 && lane == 0) {
            const uint32_t idesc = sm100::make_idesc_bf16(TM, bn);
            int s = 0, i = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++i) {
                const int b = i & 1;
                ok = mbar_wait_cluster(&acc_empty[b], ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                sm100::tc_fence_after_sync();
                const uint32_t d = tmem_base + (uint32_t)(b * BN_MAX);
                for (int ks = 0; ks < a.k_steps; ++ks) {
                    ok = sm100::mbar_wait(&full[s], ph, abort_flag);
                    if (!ok) break;
                    sm100::tc_fence_after_sync();
                    const uint32_t st = sm100::smem_u32(smem + s * stage_bytes);
                    const uint64_t da = sm100::make_desc_k_sw128(st), db = sm100::make_desc_k_sw128(st + A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk)
                        umma_pair(d, da + 2 * kk, db + 2 * kk, idesc, (ks > 0 || kk > 0) ? 1u : 0u);
                    umma_commit_pair(&empty[s]);
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit_pair(&acc_full[b]);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue: TMEM lane == token
        const int quarter = warp & 3;
        const uint32_t t_lane = tmem_base + ((uint32_t)(32 * quarter) << 16);
        int i = 0;
        for (int t = pair; t < tiles; t += pairs, ++i) {
            const int b = i & 1;
            int tm, tn;
            tile_at(t, a.tiles_m, a.tiles_n, tm, tn);
            if (!__all_sync(0xffffffffu, sm100::mbar_wait(&acc_full[b], (uint32_t)(i >> 1) & 1u, abort_flag))) break;
            sm100::tc_fence_after_sync();
            const int m = tm * TM + (int)rank * (TM / 2) + 32 * quarter + lane;
            const int n0 = tn * bn;
            const int n_end = n0 + bn < a.N ? n0 + bn : a.N;
            for (int n = n0; n < n_end; n += 32) {
                uint32_t r[32];
                sm100::tmem_ld_32x32(t_lane + (uint32_t)(b * BN_MAX + n - n0), r);
                sm100::tmem_ld_wait();
                const int cnt = n_end - n < 32 ? n_end - n : 32;
                if (m >= a.M) {
                    // a token past the end: nothing to store, the lane stays with its warp
                } else if (a.vec && cnt == 32) {
                    if (a.bias != nullptr) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __ldg(a.bias + n + j));
                    }
                    if (a.y_dtype == HXQ_F32) {
                        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<float*>(a.y) + (int64_t)m * a.ldy + n);
#pragma unroll
                        for (int j = 0; j < 8; ++j) dst[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                    } else {
                        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(a.y) + (int64_t)m * a.ldy + n);
                        uint32_t p[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) p[j] = pack16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]), a.y_dtype);
#pragma unroll
                        for (int j = 0; j < 4; ++j) dst[j] = make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (j < cnt)
                            store_from_f32(a.y, (int64_t)m * a.ldy + n + j,
                                           __uint_as_float(r[j]) + (a.bias != nullptr ? a.bias[n + j] : 0.f), a.y_dtype);
                }
                __syncwarp();
            }
            sm100::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_remote(map_to_rank(sm100::smem_u32(&acc_empty[b]), 0));
        }
    }

    sm100::tc_fence_before_sync();
    __syncwarp();
    cluster_sync();       // no CTA leaves while its pair may still signal or read it
    if (warp == 1) {
        sm100::tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    __syncwarp();
    cluster_sync();
    if (threadIdx.x == 0 && *abort_flag != 0 && a.status != nullptr) atomicExch(a.status, HXQ_E_TIMEOUT);
}

// ---- host side ---------------------------------------------------------------------

// Time of a 64-column step of a BN-wide tile, in units of 0.01 us, measured: 0.43 us at 256 columns and 0.33 at
// 64.  It follows the bytes an SM stages (16 KB of tokens whatever the width) more than the MMAs, and not the
// depth of the ring (6 and 11 stages of 64 columns take the same time).
static int step_cost(int bn) { return 30 + bn / 20; }

// Row-tile width: the multiple of 32 that needs the least (waves of tiles) x (time of a step).
static int pick_tile(int tiles_m, int N, int pairs, int64_t& best_cost) {
    int best = BN_MAX;
    best_cost = INT64_MAX;
    for (int bn = BN_MAX; bn >= 64; bn -= 32) {
        const int64_t tiles = (int64_t)tiles_m * ((N + bn - 1) / bn);
        const int64_t cost = ((tiles + pairs - 1) / pairs) * step_cost(bn);
        if (cost < best_cost) { best_cost = cost; best = bn; }
    }
    return best;
}

// Weight rows per tile of the product of M tokens and N rows.
int32_t row_tile(int32_t M, int32_t N, int n_sm) {
    int64_t cost;
    return pick_tile((M + TM - 1) / TM, N, n_sm / 2, cost);
}

// Estimated time of the product of M tokens and N rows of K columns, in units of 0.01 us.
int64_t product_cost(int32_t M, int32_t N, int32_t K, int n_sm) {
    int64_t per_step;
    pick_tile((M + TM - 1) / TM, N, n_sm / 2, per_step);
    return per_step * ((K + BK - 1) / BK);
}

// x: bf16 [M, K], row stride ldx elements; w: bf16 [ceil(K / 64)][N][64] (zeros from K on); y: column 0 of these N rows.
int run(const __nv_bfloat16* x, int64_t ldx, int32_t M, const __nv_bfloat16* w, int32_t N, int32_t K,
        const float* bias, void* y, int y_dtype, int64_t ldy, int n_sm, int32_t* status_word, cudaStream_t stream) {
    Args a;
    const int pairs = n_sm / 2;
    a.bias = bias; a.y = y; a.status = status_word; a.ldy = ldy;
    a.M = M; a.N = N; a.k_steps = (K + BK - 1) / BK;
    a.tiles_m = (M + TM - 1) / TM;
    int64_t cost;
    a.bn = pick_tile(a.tiles_m, N, pairs, cost);
    a.stages = stages_for(a.bn);
    a.tiles_n = (N + a.bn - 1) / a.bn;
    a.y_dtype = y_dtype;
    a.vec = aligned_to(y, 16) && (ldy * dtype_size(y_dtype)) % 16 == 0;
    CUtensorMap mx, mw;
    if (!gemm::make_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, (uint64_t)K, (uint64_t)M, (uint64_t)ldx * 2, BK, TM / 2,
                           CU_TENSOR_MAP_SWIZZLE_128B) ||
        !gemm::make_map_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, BK, (uint64_t)a.k_steps * N, BK * 2, BK,
                           (uint32_t)(a.bn / 2), CU_TENSOR_MAP_SWIZZLE_128B))
        return HXQ_E_DEVICE;
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(gemm_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL) != cudaSuccess)
            return HXQ_E_DEVICE;
        attr_set[dev] = true;
    }
    const int tiles = a.tiles_m * a.tiles_n;
    const int grid = 2 * (tiles < pairs ? tiles : pairs);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM_TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // set-up on SMs that the previous kernel has left
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gemm_dense_kernel, mx, mw, a) == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

}  // namespace gemmd
}  // namespace hxq

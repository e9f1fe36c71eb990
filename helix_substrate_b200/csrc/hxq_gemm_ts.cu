// hxq_gemm, 5 .. 128 tokens: y[m, o] = sum_i x[m, i] * W^[o, i] + sidecar + bias on the tensor cores
// with the dequantised weights handed to the MMA through TENSOR MEMORY, never through shared memory.
//
// At these token counts the product is still bound by the index stream (one byte and one table lookup
// per weight, each weight used for at most 128 tokens), so the kernel is built like the decode kernel,
// not like a GEMM: everything that is not a lookup is kept off the instruction stream of the warps
// that do the lookups.
//
//   * CTA tile: 128 output rows x BN tokens (BN = 16, 32, 64, 128), K walked in boxes of 128 columns, one
//     CTA per SM; small row-tile grids split K over gridDim.z (fp32 partials + a fixed-order sum).
//   * sixteen dequantising warps (2..17): four per TMEM lane quarter, ONE THREAD PER OUTPUT ROW, and each
//     of the four takes a contiguous quarter of the CTA's K range, a whole box at a time; the MMAs take
//     the quarters' boxes in turn.  So a thread does what it does once per box - scale and offset (a
//     16-byte load for four boxes), ring and barrier bookkeeping, the hand-over - once per 128 weights,
//     and a warp reads only index bytes that it copied itself.  (With the four warps of a quarter on 32
//     columns each of every box, that was paid once per 32 or 64 weights, and the boxes, copied by
//     all threads together, needed two more barriers each.)
//   * index bytes: 16-byte asynchronous copies, four lanes per row's 64 bytes, into the warp's ring of
//     three or four half boxes (2 KB each), waited for with the warp's own copy groups.
//   * per weight one byte-permute (code -> shared address) and one load from the lane-replicated codebook
//     (bank == lane); per pair one packed fp32 FMA (scale, offset) and one pack to bf16; 32 columns go
//     with one tcgen05.st 32x32b straight into the A operand's columns of tensor memory (TMEM lane ==
//     output row).  That body is kept in a loop: unrolled four times, with the sidecar's patch in each,
//     the warps' code did not fit the instruction caches (18 % of the stall cycles).
//   * sidecar: a thread-local cursor; a box's entries are patched in tensor memory when the box is
//     complete.  (Adding the sidecar term in the epilogue instead - delta times the activation at its
//     column, per token - was tried: every such load is a cache-line look-up per lane, 13 us per tile at
//     32 tokens and 44 us at 128.)
//   * warp 0, one lane: TMA producer of the activation tiles (two 64-column boxes of bf16 per step,
//     128-byte swizzled, ring of two to four).  No multicast, no cluster.
//   * warp 1, one lane: issues tcgen05.mma kind::f16 with A from tensor memory and B (activations,
//     K-major, 128-byte swizzle) from shared memory into the fp32 accumulator in tensor memory, and
//     commits the stage, which frees its activation tile and its A columns.
//   * epilogue (the dequantising warps): accumulator -> registers, + bias, store.
//
// Launched dependent (griddepcontrol): the table, the first index boxes and the cursors are set up while
// the previous kernel drains, where it leaves SMs free.
//
// Measured (us, graph replay, this layout / the one of 32-column slices and shared boxes):
//   tokens                        5           32          64          128
//   gate [18944 x 3584]           28.9 / 39.5 29.3 / 39.4 30.1 / 39.4 32.0 / 46.9
//   down [3584 x 18944], K split  40.5 / 47.9 40.3 / 48.0 41.7 / 48.6 44.2 / 58.8
//   q [3584 x 3584], K split      15.8 / 18.6 16.1 / 19.1 18.0 / 19.7 20.3 / 24.5
// Bound by the instruction stream: 8 warp instructions per 32 weights at 54 % issue.
//
// Every mbarrier wait is clock-bounded; a wait that gives up raises a CTA-wide abort flag and the
// global status word (HXQ_E_TIMEOUT); every other wait of the CTA then returns at its next poll,
// in-flight copies are waited for and tensor memory is freed before the CTA returns.

#include <cuda.h>
#include <stdlib.h>

#include "hxq_common.cuh"
#include "hxq_sm100.cuh"

namespace hxq {
namespace gemm {   // helpers shared with the large-token kernel (hxq_gemm.cu)
bool make_map_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t outer,
                 uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw);
void launch_splitk_reduce(const float* partial, int splits, int M, int out_features, const float* bias, void* y,
                          int y_dtype, int64_t ldy, cudaStream_t stream);
}  // namespace gemm

namespace gemmts {

constexpr int BM = 128;             // output rows per CTA = UMMA M = TMEM lanes
constexpr int KS = 128;             // K columns per box: one step of the MMAs
constexpr int DEQ_WARPS = 16;       // four warps per TMEM lane quarter, each takes whole boxes of its own quarter of K
constexpr int NUM_THREADS = 32 * (2 + DEQ_WARPS);   // activation producer, MMA issuer, 16 dequantisers
constexpr int LUT_BYTES = 256 * 256;            // entry c, lane l at c * 256 + l * 4, base on a 64 KB boundary
constexpr int SMEM_TOTAL = 232448;
constexpr int TMEM_COLS = 512;
constexpr int A_COLS = KS / 2;                  // 64 columns of packed bf16 pairs per box

struct Args {
    const float* cb;
    const void* scales;
    const void* offsets;
    const int32_t* rowptr;
    const int32_t* cols;
    const float* deltas;
    const float* bias;
    const uint8_t* idx;        // index matrix [out_features, ld_idx]
    int64_t ld_idx;
    void* y;
    int32_t* status;
    float* partial;            // [splits][M][out_features] when the K range is split, else nullptr
    int64_t ldy;
    int32_t out_features, in_features, col0, group_size, ld_st, st_dtype, n_groups;
    int32_t M, y_dtype, k_steps, k_per_split;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));   // first source -> upper half
    return r;
}

// D[tmem] (+)= A[tmem] * B[smem], bf16 x bf16 -> fp32, issued by ONE thread.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 registers per thread -> 16 consecutive columns of this thread's TMEM lane (whole warp).
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// One bf16 half of a packed pair += delta (the value is re-rounded to bf16).
__device__ __forceinline__ uint32_t add_to_half(uint32_t pair, int hi, float delta) {
    const float v = __uint_as_float(hi ? (pair & 0xffff0000u) : (pair << 16)) + delta;
    const uint32_t b = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
    return hi ? ((pair & 0x0000ffffu) | (b << 16)) : ((pair & 0xffff0000u) | b);
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// Two neighbouring lookups of one index word as a packed pair (see hxq_gemv.cu).
__device__ __forceinline__ uint64_t lut_pair(uint32_t word, uint32_t lane_key, int k0) {
    const uint32_t a0 = __byte_perm(word, lane_key, 0x7604u | (uint32_t)(k0 << 4));
    const uint32_t a1 = __byte_perm(word, lane_key, 0x7604u | (uint32_t)((k0 + 1) << 4));
    uint64_t r;
    asm volatile("{\n\t.reg .f32 lo, hi;\n\tld.shared.f32 lo, [%1];\n\tld.shared.f32 hi, [%2];\n\t"
                 "mov.b64 %0, {lo, hi};\n\t}" : "=l"(r) : "r"(a0), "r"(a1));
    return r;
}
// bf16x2(c0 * s + t, c1 * s + t): one packed fp32 FMA, each half rounded like fmaf.
__device__ __forceinline__ uint32_t affine_pack(uint64_t c, uint64_t s2, uint64_t t2) {
    uint32_t r;
    asm("{\n\t.reg .b64 v;\n\t.reg .f32 lo, hi;\n\t"
        "fma.rn.f32x2 v, %1, %2, %3;\n\tmov.b64 {lo, hi}, v;\n\t"
        "cvt.rn.bf16x2.f32 %0, hi, lo;\n\t}" : "=r"(r) : "l"(c), "l"(s2), "l"(t2));
    return r;
}
__device__ __forceinline__ uint64_t twice(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

// Per token tile: NB activation tiles, NA A-operand slots (64 columns each) and R half boxes per
// dequantising warp.  The table sits on a 64 KB boundary of the shared window, which leaves ~63 KB
// below and 100 KB above it: the activation tiles go below while they fit, then above, the warps'
// rings into what is left.
template <int BN> struct Rings;
template <> struct Rings<16> { static constexpr int NB = 4, NA = 7, R = 4; };
template <> struct Rings<32> { static constexpr int NB = 3, NA = 7, R = 4; };
template <> struct Rings<64> { static constexpr int NB = 3, NA = 7, R = 3; };
template <> struct Rings<128> { static constexpr int NB = 2, NA = 6, R = 3; };
constexpr int HALF_BYTES = 32 * 64;         // a warp's half box: 32 rows x 64 codes

template <int BN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_ts_kernel(const __grid_constant__ CUtensorMap map_x, const Args a) {
    constexpr int B_BYTES = BN * KS * 2;                 // two [BN x 64] bf16 sub-tiles
    constexpr int NB = Rings<BN>::NB, NA = Rings<BN>::NA, R = Rings<BN>::R;
    constexpr uint32_t RING = R * HALF_BYTES;
    static_assert((BN < 32 ? 32 : BN) + NA * A_COLS <= TMEM_COLS, "accumulator + A ring must fit tensor memory");
    static_assert(NB <= 8 && NA <= 8, "barrier layout");
    extern __shared__ __align__(1024) char smem_raw[];
    const uint32_t smem_base = sm100::smem_u32(smem_raw);
    const uint32_t lut_base = (smem_base + 0xFFFFu) & ~0xFFFFu;
    char* lut = smem_raw + (lut_base - smem_base);
    const uint32_t lo0 = (smem_base + 1023u) & ~1023u;
    const uint32_t hi0 = lut_base + LUT_BYTES;
    const int fit = (int)(lut_base - lo0) / B_BYTES;
    const int nb_lo = fit < NB ? fit : NB;                                   // activation tiles below the table
    auto b_slot = [&](int i) -> uint32_t { return i < nb_lo ? lo0 + (uint32_t)(i * B_BYTES) : hi0 + (uint32_t)((i - nb_lo) * B_BYTES); };
    const uint32_t lo1 = lo0 + (uint32_t)(nb_lo * B_BYTES), hi1 = hi0 + (uint32_t)((NB - nb_lo) * B_BYTES);
    const int nr_lo = (int)((lut_base - lo1) / RING) < DEQ_WARPS ? (int)((lut_base - lo1) / RING) : DEQ_WARPS;   // warps' rings below it
    const bool layout_ok = hi1 + (uint32_t)(DEQ_WARPS - nr_lo) * RING <= smem_base + SMEM_TOTAL;
    // barriers live in the unused upper halves of the table's first rows
    uint64_t* b_full = reinterpret_cast<uint64_t*>(lut + 128);            // [NB] activation tile landed
    uint64_t* b_free = b_full + 8;                                        // [NB] MMAs that read it retired
    uint64_t* a_full = reinterpret_cast<uint64_t*>(lut + 256 + 128);      // [NA] A columns of the box written
    uint64_t* a_free = a_full + 8;                                        // [NA] MMAs that read them retired
    uint64_t* acc_full = reinterpret_cast<uint64_t*>(lut + 512 + 128);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BN;
    const int o0 = blockIdx.y * BM;
    // this CTA's boxes [KS0, KS0 + NK), in four contiguous parts, one per group of four warps; the
    // MMAs take the parts' boxes in turn: step i is box i / 4 of part i % 4
    const int KS0 = blockIdx.z * a.k_per_split;
    const int NK = (a.k_steps - KS0 < a.k_per_split) ? a.k_steps - KS0 : a.k_per_split;
    auto part_first = [&](int q) -> int { return KS0 + q * (NK >> 2) + (q < (NK & 3) ? q : (NK & 3)); };

    // ---- the dequantising warps (2..17; the definitions below are only used by them)
    const int dw = warp - 2;
    const int quarter = warp & 3;                 // TMEM lanes this warp may touch: [32 * quarter, +32)
    const int kq = dw >> 2;                       // its part of the K range (warps 2..17: every quarter gets 0..3 once)
    const int row = o0 + 32 * quarter + lane;     // this thread's output row
    const bool row_ok = row < a.out_features;
    const bool affine = a.group_size > 0;
    const int box0 = part_first(kq);
    const int n_box = (NK >> 2) + (kq < (NK & 3) ? 1 : 0);
    const int n_half = 2 * n_box;
    const uint32_t ring = dw < nr_lo ? lo1 + (uint32_t)dw * RING : hi1 + (uint32_t)(dw - nr_lo) * RING;

    // ---- index copies: a warp copies the 32 x 64 half boxes that it reads itself, four lanes per
    // row's 64 bytes, eight rows per instruction; 16-byte piece c of row r at r * 64 + (c ^ (r / 2 & 3)) * 16,
    // so that eight lanes reading the same piece of their own rows meet no bank twice
    const int c_row = lane >> 2, c_piece = lane & 3;
    const uint32_t c_dst = (uint32_t)(c_row * 64 + ((c_piece ^ ((c_row >> 1) & 3)) << 4));   // (row + 8 has the same swizzle)
    const int c_rows = a.out_features - (o0 + 32 * quarter + c_row);        // rows of this lane's column that exist, by eight
    const int64_t c_k0 = (int64_t)box0 * KS + c_piece * 16;
    const uint8_t* c_src = a.idx + (int64_t)(c_rows > 0 ? o0 + 32 * quarter + c_row : 0) * a.ld_idx + c_k0;
    auto copy_half = [&](int q, uint32_t slot) {      // half box q of this warp; always one group
        if (q < n_half) {
            const bool in_k = c_k0 + 64 * q < a.in_features;       // (in_features is a multiple of 16)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // rows past the matrix and columns past its end are filled with zeros (source size 0)
                const uint32_t n = (in_k && 8 * i < c_rows) ? 16u : 0u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                             :: "r"(ring + slot + c_dst + (uint32_t)(i * 512)), "l"(n ? c_src + 64 * q + (int64_t)(8 * i) * a.ld_idx : a.idx), "r"(n) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NB; ++s) {
            sm100::mbar_init(&b_full[s], 1);
            sm100::mbar_init(&b_free[s], 1);
        }
        for (int s = 0; s < NA; ++s) {
            sm100::mbar_init(&a_full[s], 4);
            sm100::mbar_init(&a_free[s], 1);
        }
        sm100::mbar_init(acc_full, 1);
        *abort_flag = 0;
        sm100::fence_barrier_init();
        sm100::prefetch_tensormap(&map_x);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // The first half boxes are asked for before the rest is set up: the table build and the
    // tensor-memory allocation below overlap their flight.
    if (layout_ok && warp >= 2) {
#pragma unroll
        for (int q = 0; q < R - 1; ++q) copy_half(q, (uint32_t)(q * HALF_BYTES));
    }
    if (warp == 1) {
        sm100::tmem_alloc(tmem_slot, TMEM_COLS);
        sm100::tmem_relinquish();
    }
    // lane-replicated codebook (the lower 128 bytes of each 256-byte row), a warp's entries all asked for at once
    {
        constexpr int PER = (256 + NUM_THREADS / 32 - 1) / (NUM_THREADS / 32);
        float c[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) c[j] = warp + j * (NUM_THREADS / 32) < 256 ? a.cb[warp + j * (NUM_THREADS / 32)] : 0.f;
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (warp + j * (NUM_THREADS / 32) < 256) *reinterpret_cast<float*>(lut + (warp + j * (NUM_THREADS / 32)) * 256 + lane * 4) = c[j];
    }
    // ---- sidecar cursor of this thread's row inside its part of K: entries are sorted by column; the next two are
    // held, so that the load that refills them is not waited for when one is used.  Started here, in the shadow
    // of the first boxes' flight, and with the last 16 candidates in one round of loads: a chain of
    // dependent cache misses down to one entry held every CTA up for 4 us before its first lookup.
    int e_cur = 0, e_end = 0, nc = 0x7fffffff, nc1 = 0x7fffffff;
    float nd = 0.f, nd1 = 0.f;
    if (layout_ok && warp >= 2 && a.rowptr != nullptr && row_ok && n_half > 0) {
        e_cur = a.rowptr[row];
        e_end = a.rowptr[row + 1];
        if (box0 > 0) {
            const int k0 = box0 * KS;
            int hi = e_end;
            while (hi - e_cur > 16) {
                const int mid = (e_cur + hi) >> 1;
                if (a.cols[mid] < k0) e_cur = mid + 1; else hi = mid;
            }
            int below = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) below += (e_cur + j < hi && a.cols[e_cur + j] < k0) ? 1 : 0;
            e_cur += below;
        }
        if (e_cur < e_end) { nc = a.cols[e_cur]; nd = a.deltas[e_cur]; }
        if (e_cur + 1 < e_end) { nc1 = a.cols[e_cur + 1]; nd1 = a.deltas[e_cur + 1]; }
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    sm100::tc_fence_after_sync();
    // everything above reads weights only; activations, results and partials belong to the stream's earlier kernels until here
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a0 = tmem_base + (uint32_t)(BN < 32 ? 32 : BN);   // the A ring follows the accumulator's columns

    if (!layout_ok) {
        if (threadIdx.x == 0 && a.status != nullptr) atomicExch(a.status, HXQ_E_SHAPE);
    } else if (warp == 0) {
        // ------------------------------------------------------------ activation producer (TMA)
        if (lane == 0) {
            int armed = 0;
            for (int i = 0; i < NK; ++i) {
                const int s = i % NB;
                if (!sm100::mbar_wait(&b_free[s], ((uint32_t)(i / NB) & 1u) ^ 1u, abort_flag, 2000000000LL, 100u)) break;
                char* bt = smem_raw + (b_slot(s) - smem_base);
                const int k = (part_first(i & 3) + (i >> 2)) * KS;
                sm100::mbar_arrive_expect_tx(&b_full[s], (uint32_t)B_BYTES);
#pragma unroll
                for (int j = 0; j < 2; ++j)           // 64-column sub-tiles
                    sm100::tma_load_2d(bt + j * (BN * 128), &map_x, &b_full[s], k + 64 * j, m0);
                armed = i + 1;
            }
            if (*abort_flag != 0) {
                for (int i = (armed > NB ? armed - NB : 0); i < armed; ++i)
                    sm100::mbar_wait(&b_full[i % NB], (uint32_t)(i / NB) & 1u, abort_flag, 200000000LL);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            constexpr uint32_t idesc = sm100::make_idesc_bf16(BM, BN);
            bool ok = true;
            for (int i = 0; i < NK && ok; ++i) {
                const int s = i % NB, sa = i % NA;
                ok = sm100::mbar_wait(&b_full[s], (uint32_t)(i / NB) & 1u, abort_flag, 2000000000LL, 50u) &&
                     sm100::mbar_wait(&a_full[sa], (uint32_t)(i / NA) & 1u, abort_flag, 2000000000LL, 50u);
                if (!ok) break;
                sm100::tc_fence_after_sync();
                // B: sub-tile kk / 4 (64 K columns each), + 32 bytes (2 in descriptor units) per 16-column slice
                const uint64_t db0 = sm100::make_desc_k_sw128(b_slot(s));
                const uint32_t ta = tmem_a0 + (uint32_t)(sa * A_COLS);
#pragma unroll
                for (int kk = 0; kk < KS / 16; ++kk) {
                    const uint64_t db = db0 + (uint64_t)((kk >> 2) * (BN * 128 / 16) + 2 * (kk & 3));
                    umma_bf16_ts(tmem_base, ta + (uint32_t)(kk * 8), db, idesc, (i > 0 || kk > 0) ? 1u : 0u);
                }
                sm100::umma_commit(&b_free[s]);
                sm100::umma_commit(&a_free[sa]);
            }
            if (ok) sm100::umma_commit(acc_full);
        }
    } else {
        // ------------------------------------------------------------ dequantising warps
        const uint32_t lane_key = lut_base | ((uint32_t)lane << 2);
        const uint32_t t_row = tmem_a0 + ((uint32_t)(32 * quarter) << 16);
        const uint32_t r_src = ring + (uint32_t)(lane * 64);
        const uint32_t r_swz = (uint32_t)((lane >> 1) & 3);

        // ---- scale / offset of this thread's row, one pair per half box (group_size and col0 are multiples of 64).
        // Block case (128-column groups, fp32 tables with 16-byte aligned rows, shard starting on a group - every
        // Qwen2.5 shape): one 16-byte load each for four boxes, a block ahead; else one pair, a half box ahead.
        const int g_base = affine ? a.col0 / a.group_size : 0;
        const bool st_block = affine && a.group_size == KS && a.col0 % KS == 0 && a.st_dtype == HXQ_F32 && a.ld_st % 4 == 0 &&
                              ((reinterpret_cast<uintptr_t>(a.scales) | reinterpret_cast<uintptr_t>(a.offsets)) & 15) == 0;
        const int64_t st_row = (int64_t)(row_ok ? row : 0) * a.ld_st;
        auto load_block = [&](int blk, float4& s4, float4& t4) {      // groups 4 blk .. 4 blk + 3
            s4 = make_float4(1.f, 1.f, 1.f, 1.f); t4 = make_float4(0.f, 0.f, 0.f, 0.f);
            const int n = a.n_groups - 4 * blk;
            const float* ps = reinterpret_cast<const float*>(a.scales) + st_row + 4 * blk;
            const float* pt = reinterpret_cast<const float*>(a.offsets) + st_row + 4 * blk;
            if (n >= 4) {
                s4 = *reinterpret_cast<const float4*>(ps);
                t4 = *reinterpret_cast<const float4*>(pt);
            } else if (n > 0) {     // last, short block of the row: never past the row's groups
                s4.x = ps[0]; t4.x = pt[0];
                if (n > 1) { s4.y = ps[1]; t4.y = pt[1]; }
                if (n > 2) { s4.z = ps[2]; t4.z = pt[2]; }
            }
        };
        auto load_st = [&](int q, float& s, float& t) {               // half box q of this warp
            s = 1.f; t = 0.f;
            if (affine) {
                int g = (a.col0 + box0 * KS + 64 * q) / a.group_size - g_base;
                g = g < a.n_groups ? g : a.n_groups - 1;      // K tail: those activations are zero
                const int64_t o = st_row + g;
                if (a.st_dtype == HXQ_F32) {
                    s = reinterpret_cast<const float*>(a.scales)[o];
                    t = reinterpret_cast<const float*>(a.offsets)[o];
                } else {
                    s = __half2float(reinterpret_cast<const __half*>(a.scales)[o]);
                    t = __half2float(reinterpret_cast<const __half*>(a.offsets)[o]);
                }
            }
        };
        float4 s4 = make_float4(1.f, 1.f, 1.f, 1.f), t4 = make_float4(0.f, 0.f, 0.f, 0.f), s4n = s4, t4n = t4;
        float sc_n = 1.f, of_n = 0.f;
        if (n_half > 0) {
            if (st_block) load_block(box0 >> 2, s4n, t4n);
            else load_st(0, sc_n, of_n);
        }

        bool failed = false;          // one of this thread's bounded waits gave up (or saw the abort flag)
        uint32_t slot = 0;
        for (int j = 0; j < n_box; ++j) {
            const int i = 4 * j + kq;             // the step this box is
            const int sa = i % NA;
            const uint32_t t_dst = t_row + (uint32_t)(sa * A_COLS);
            if (st_block) {
                const int g = box0 + j;
                if (j == 0 || (g & 3) == 0) {
                    s4 = s4n; t4 = t4n;
                    if (((g >> 2) + 1) * 4 < box0 + n_box) load_block((g >> 2) + 1, s4n, t4n);
                }
                sc_n = (g & 3) == 0 ? s4.x : ((g & 3) == 1 ? s4.y : ((g & 3) == 2 ? s4.z : s4.w));
                of_n = (g & 3) == 0 ? t4.x : ((g & 3) == 1 ? t4.y : ((g & 3) == 2 ? t4.z : t4.w));
            }
            float sc = 1.f, of = 0.f;
            // 32 columns at a time, NOT unrolled: with the four bodies side by side the eighteen warps' code did not fit
            // the instruction caches, a fifth of all stall cycles
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                if ((c & 1) == 0) {
                    const int q = 2 * j + (c >> 1);
                    asm volatile("cp.async.wait_group %0;" :: "n"(R - 2) : "memory");
                    __syncwarp();     // half box q has landed for every lane, and every lane has half box q - 1 in registers
                    copy_half(q + R - 1, slot == 0 ? RING - HALF_BYTES : slot - HALF_BYTES);     // into the slot half box q - 1 had
                    sc = sc_n; of = of_n;
                    if (!st_block && q + 1 < n_half) load_st(q + 1, sc_n, of_n);
                }
                uint32_t w[8];
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(w[4 * k]), "=r"(w[4 * k + 1]), "=r"(w[4 * k + 2]), "=r"(w[4 * k + 3])
                                 : "r"(r_src + slot + (((2 * (c & 1) + k) ^ r_swz) << 4)) : "memory");
                if (c & 1) slot = slot + HALF_BYTES == RING ? 0 : slot + HALF_BYTES;
                const uint64_t s2 = twice(sc), t2 = twice(of);
                uint32_t out[16];
#pragma unroll
                for (int p = 0; p < 16; ++p)
                    out[p] = affine_pack(lut_pair(w[p >> 1], lane_key, 2 * (p & 1)), s2, t2);
                if (c == 0) {
                    // the slot's columns are free once the MMAs that read them NA steps ago have retired
                    // (warp-uniform outcome: the store below is a whole-warp instruction)
                    if (i >= NA && !__all_sync(0xffffffffu, sm100::mbar_wait(&a_free[sa], (uint32_t)(i / NA - 1) & 1u, abort_flag))) {
                        failed = true;
                        break;
                    }
                    sm100::tc_fence_after_sync();
                }
                tmem_st_32x16(t_dst + (uint32_t)(16 * c), out);
            }
            if (failed) break;
            tmem_st_wait();
            // sidecar entries of these 32 rows inside the box: column by column, read back, patched in the lanes that
            // have an entry there, and stored again (about four rounds per box at 0.1 %).  A jump into the packed
            // registers per entry diverged once per entry and chunk and carried sixteen bodies per chunk.
            const int k_lo = (box0 + j) * KS;
            for (uint32_t m; (m = __ballot_sync(0xffffffffu, nc < k_lo + KS)) != 0u; ) {
                const int col = __shfl_sync(0xffffffffu, (nc - k_lo) >> 1, __ffs(m) - 1);
                uint32_t v;
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(t_dst + (uint32_t)col) : "memory");
                sm100::tmem_ld_wait();
                if (nc < k_lo + KS && ((nc - k_lo) >> 1) == col) {
                    v = add_to_half(v, nc & 1, nd);
                    ++e_cur;
                    nc = nc1; nd = nd1;
                    if (e_cur + 1 < e_end) { nc1 = a.cols[e_cur + 1]; nd1 = a.deltas[e_cur + 1]; } else { nc1 = 0x7fffffff; }
                }
                __syncwarp();
                asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(t_dst + (uint32_t)col), "r"(v) : "memory");
                tmem_st_wait();
            }
            sm100::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&a_full[sa]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // (a loop left early must not retire with copies in flight)

        // ------------------------------------------------------------ epilogue
        // the four warps of a quarter split the token columns
        {
            constexpr int COLS_PER_WARP = BN / 4 < 8 ? 8 : BN / 4;   // 8, 16 or 32 (16 tokens: two of the four warps)
            const int c_lo = kq * COLS_PER_WARP;
            if (!failed && c_lo < BN && sm100::mbar_wait(acc_full, 0u, abort_flag)) {
                sm100::tc_fence_after_sync();
                float* part = a.partial ? a.partial + (int64_t)blockIdx.z * a.M * a.out_features : nullptr;
                const float bias = (a.bias != nullptr && row_ok && part == nullptr) ? a.bias[row] : 0.f;
#pragma unroll 1
                for (int c0 = c_lo; c0 < c_lo + COLS_PER_WARP; c0 += 8) {
                    if (m0 + c0 >= a.M) break;           // warp-uniform
                    uint32_t v[8];
                    __syncwarp();
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                        : "r"(tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)c0)
                        : "memory");
                    sm100::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int m = m0 + c0 + j;
                        if (row_ok && m < a.M) {
                            const float acc = __uint_as_float(v[j]);
                            if (part != nullptr) part[(int64_t)m * a.out_features + row] = acc;
                            else store_from_f32(a.y, (int64_t)m * a.ldy + row, acc + bias, a.y_dtype);
                        }
                    }
                }
            }
        }
    }

    sm100::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        sm100::tc_fence_after_sync();
        sm100::tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag == 1 && a.status != nullptr) atomicExch(a.status, HXQ_E_TIMEOUT);
}

}  // namespace gemmts
}  // namespace hxq

namespace hxq {
namespace gemmts {

// ---- host side ---------------------------------------------------------------------

static int sm_count() {      // asked once per device
    static int cached[64] = {0};
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return n_sm;
    if (cached[dev] == 0)
        cached[dev] = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n_sm > 0 ? n_sm : 148;
    return cached[dev];
}

static int pick_bn(int M) { return M > 64 ? 128 : (M > 32 ? 64 : (M > 16 ? 32 : 16)); }

// K slices per output tile: enough CTAs to fill the GPU when the row-tile grid alone does not, at
// least four boxes (512 columns) each.  k_boxes: 128-column boxes of the K range.
static int pick_splits(int grid_m, int grid_o, int k_boxes, int n_sm) {
    const int tiles = grid_m * grid_o;
    if (tiles * 2 > n_sm) return 1;
    int s = n_sm / tiles;
    if (s > 8) s = 8;
    if (s > k_boxes / 4) s = k_boxes / 4;
    return s < 1 ? 1 : s;
}

// Largest token count this kernel takes (128); HXQ_GEMM_TS_MAX_M lowers it (0 = never) for A/B timing.
static int max_tokens() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("HXQ_GEMM_TS_MAX_M");
        int n = e ? atoi(e) : 128;
        v = n < 0 ? 0 : (n > 128 ? 128 : n);
    }
    return v;
}

bool covers(const hxq_desc* d, int32_t M) {
    return M >= 1 && M <= max_tokens() && (d->in_features % 16 == 0) && (d->ld_idx % 16 == 0) && aligned_to(d->indices, 16) &&
           (d->col0 % 64 == 0) && (d->group_size == 0 || d->group_size % 64 == 0);
}

size_t split_bytes(const hxq_desc* d, int32_t M) {
    const int BN = pick_bn(M);
    const int s = pick_splits((M + BN - 1) / BN, (d->out_features + BM - 1) / BM, (d->in_features + KS - 1) / KS, sm_count());
    return s > 1 ? (size_t)s * M * d->out_features * sizeof(float) : 0;
}

template <int BN>
static int launch(const CUtensorMap& mx, const Args& a, int grid_m, int grid_o, int splits, cudaStream_t stream) {
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(gemm_ts_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL) != cudaSuccess)
            return HXQ_E_DEVICE;
        attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_m, grid_o, splits);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM_TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // set-up on SMs that the previous kernel has left
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_weights_on_stream ? 0 : 1;   // weights still being written on this stream: no early start
    return cudaLaunchKernelEx(&cfg, gemm_ts_kernel<BN>, mx, a) == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

// xb: the activations as bf16 with a 16-byte aligned row stride (the caller converted them if needed);
// split_ws: room for the fp32 partials (split_bytes) or nullptr.
int run(const hxq_desc* d, const __nv_bfloat16* xb, int64_t ldxb, int32_t M, void* y, int y_dtype, int64_t ldy,
        void* split_ws, size_t split_ws_bytes, int32_t* status_word, cudaStream_t stream) {
    const int BN = pick_bn(M);
    CUtensorMap mx;
    if (!gemm::make_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, xb, (uint64_t)d->in_features, (uint64_t)M,
                           (uint64_t)ldxb * 2, 64, (uint32_t)BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return HXQ_E_DEVICE;
    Args a;
    a.cb = d->codebook; a.scales = d->scales; a.offsets = d->offsets;
    a.rowptr = d->rowptr; a.cols = d->cols; a.deltas = d->deltas; a.bias = d->bias;
    a.idx = d->indices; a.ld_idx = d->ld_idx;
    a.y = y; a.status = status_word; a.ldy = ldy;
    a.out_features = d->out_features; a.in_features = d->in_features; a.col0 = d->col0;
    a.group_size = d->group_size; a.ld_st = d->ld_st; a.st_dtype = d->st_dtype;
    a.n_groups = d->group_size > 0 ? (d->col0 + d->in_features - 1) / d->group_size - d->col0 / d->group_size + 1 : 0;
    a.M = M; a.y_dtype = y_dtype;
    a.k_steps = (d->in_features + KS - 1) / KS;
    const int grid_o = (d->out_features + BM - 1) / BM;
    const int grid_m = (M + BN - 1) / BN;
    int splits = pick_splits(grid_m, grid_o, a.k_steps, sm_count());
    a.k_per_split = a.k_steps;
    a.partial = nullptr;
    if (splits > 1 && split_ws && aligned_to(split_ws, 16) &&
        split_ws_bytes >= (size_t)splits * M * d->out_features * sizeof(float)) {
        a.k_per_split = (a.k_steps + splits - 1) / splits;
        splits = (a.k_steps + a.k_per_split - 1) / a.k_per_split;   // no empty slice
        if (splits > 1) a.partial = reinterpret_cast<float*>(split_ws);
        else a.k_per_split = a.k_steps;                             // one slice after rounding: nothing to split
    } else {
        splits = 1;
    }
    int st;
    if (BN == 128) st = launch<128>(mx, a, grid_m, grid_o, splits, stream);
    else if (BN == 64) st = launch<64>(mx, a, grid_m, grid_o, splits, stream);
    else if (BN == 32) st = launch<32>(mx, a, grid_m, grid_o, splits, stream);
    else st = launch<16>(mx, a, grid_m, grid_o, splits, stream);
    if (st != HXQ_OK || splits == 1) return st;
    gemm::launch_splitk_reduce(a.partial, splits, M, d->out_features, d->bias, y, y_dtype, ldy, stream);
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

}  // namespace gemmts
}  // namespace hxq

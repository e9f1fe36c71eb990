// hxq_dequant: compressed rows -> dense fp32 / bf16 / fp16 rows.
//
// Bound by HBM writes (4 B or 2 B out per 1 B of index in).  fp32 output is
// bit-exact with the reference reader: codebook gather, optional affine with
// two roundings, then the sidecar VALUE overwrites the entry.

#include "hxq_common.cuh"

namespace hxq {

struct DequantArgs {
    const uint8_t* idx;
    const float* cb;
    const void* scales;
    const void* offsets;
    const int32_t* rowptr;
    const int32_t* cols;
    const float* values;    // nullptr: W^ + deltas
    const float* deltas;
    void* out;
    int64_t ld_idx;
    int64_t ld_out;
    int32_t row0, row1, in_features, col0, group_size, ld_st, st_dtype;
    int32_t wide;           // out rows can take 32-byte stores
    int32_t k_pad;          // columns written per row (blocked layout: in_features rounded up to 64, zeros behind)
};

// Element offset of (row lr of this call, column col).  Blocked: [column / 64][row][64], so that any rows of
// one 64-column step of the dense product are one contiguous piece of memory.
template <bool BLK>
__device__ __forceinline__ int64_t out_at(const DequantArgs& a, int lr, int col) {
    return BLK ? ((int64_t)(col >> 6) * (a.row1 - a.row0) + lr) * 64 + (col & 63) : (int64_t)lr * a.ld_out + col;
}

__device__ __forceinline__ float weight_at(const DequantArgs& a, const float* cb_s, int row, int col,
                                           uint32_t code) {
    float w = cb_s[code];
    if (a.group_size > 0) {
        int g = (a.col0 + col) / a.group_size - a.col0 / a.group_size;
        int64_t o = (int64_t)row * a.ld_st + g;
        float s = load_as_f32(a.scales, o, a.st_dtype);
        float t = load_as_f32(a.offsets, o, a.st_dtype);
        w = affine_2round(w, s, t);
    }
    return w;
}

// What a sidecar entry puts at its place: the stored value, or (values == nullptr) the reconstructed weight
// plus the delta, which is what a product adds.
__device__ __forceinline__ float sidecar_value(const DequantArgs& a, int row, int col, int e) {
    return a.values != nullptr ? a.values[e]
                               : weight_at(a, a.cb, row, col, a.idx[(int64_t)row * a.ld_idx + col]) + a.deltas[e];
}
template <bool BLK>
__device__ __forceinline__ void sidecar_entry(const DequantArgs& a, int lr, int col, float v, int out_dt) {
    store_from_f32(a.out, out_at<BLK>(a, lr, col), v, out_dt);
}
template <bool BLK>
__device__ __forceinline__ void sidecar_row(const DequantArgs& a, int lr, int lane, int out_dt) {
    const int row = a.row0 + lr;
    const int e1 = a.rowptr[row + 1];
    for (int e = a.rowptr[row] + lane; e < e1; e += 32) sidecar_entry<BLK>(a, lr, a.cols[e], sidecar_value(a, row, a.cols[e], e), out_dt);
}

// 32 bytes in one store: whole sectors, where two 16-byte stores a warp apart write each sector by halves.
__device__ __forceinline__ void st_global_32(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// Vector path.  One byte in and two or four out per weight; what bounds it is latency, so warps work alone:
// a unit is one row's run of at most 256 16-column pieces (or a few short rows), a lane takes a piece at a
// time, four asked for before the first is used, and when the unit is written the same warp puts the
// sidecar entries of its columns on top (a warp barrier orders it), their loads issued early.
// (Blocks that took runs of rows together waited for each other and for the sidecar's chain of loads
// once per run: 44 us for 18944 x 3584 to bf16; a second launch for the sidecar: 50 us.  This: 38 us, 5.3 TB/s.)
//
// * the codebook is replicated per lane (entry c, lane l at c * 256 + l * 4: bank == lane, where one copy of
//   256 floats had a warp's lookups meet in a bank three to four at a time), and a lookup's offset is one
//   byte-permute of the code word;
// * 32-byte stores where rows allow it: whole sectors, half the store instructions.
constexpr int kVecThreads = 512;
constexpr int kVecLutBytes = 256 * 256;
constexpr int kUnitPieces = 256;

template <int OUT_DT, int STM, bool BLK>
__global__ void __launch_bounds__(kVecThreads, 2)
dequant_vec_kernel(const DequantArgs a, const int rows_per_unit, const int segs, const int group_shift, const uint32_t div_magic) {
    extern __shared__ __align__(256) char lut[];
    // Only the two-pass product lets the next kernel in early: its product waits.  What follows hxq_dequant may take
    // `out` for a long-lived weight and read it before its own wait.
    if constexpr (BLK) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        constexpr int PER = 256 / (kVecThreads / 32);
        float c[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) c[j] = a.cb[warp * PER + j];
#pragma unroll
        for (int j = 0; j < PER; ++j) *reinterpret_cast<float*>(lut + (warp * PER + j) * 256 + lane * 4) = c[j];
    }
    if constexpr (BLK) asm volatile("griddepcontrol.wait;" ::: "memory");      // (the scratch may still be read by the product before this one)
    __syncthreads();
    const uint32_t lane4 = (uint32_t)lane << 2;
    const uint32_t vec_per_row = (uint32_t)a.k_pad >> 4;
    const int n_rows = a.row1 - a.row0;
    const int g_base = STM ? a.col0 / a.group_size : 0;
    const int seg_pieces = (vec_per_row + segs - 1) / segs;
    const int64_t units = (int64_t)((n_rows + rows_per_unit - 1) / rows_per_unit) * segs;

    for (int64_t unit = (int64_t)blockIdx.x * (kVecThreads / 32) + warp; unit < units; unit += (int64_t)gridDim.x * (kVecThreads / 32)) {
        const int ru = (int)(unit / segs), seg = (int)(unit - (int64_t)ru * segs);
        const int lr0 = ru * rows_per_unit;
        const int nr = n_rows - lr0 < rows_per_unit ? n_rows - lr0 : rows_per_unit;
        const uint32_t first = (uint32_t)(seg * seg_pieces);
        const uint32_t total = segs > 1 ? (first + seg_pieces < vec_per_row ? first + seg_pieces : vec_per_row) : (uint32_t)nr * vec_per_row;
        // sidecar of the unit's (first) row: this lane's entry
        int e0 = 0, e1 = 0, sc_col = -1;
        float sc_val = 0.f;
        if (a.rowptr != nullptr) { e0 = a.rowptr[a.row0 + lr0]; e1 = a.rowptr[a.row0 + lr0 + 1]; }
        constexpr int U = 4;
        for (uint32_t v0 = first + lane; v0 - lane < total; v0 += 32 * U) {
            uint4 q[U];
            float s[U], t[U];
            int lr[U], col[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t v = v0 + 32 * u;
                lr[u] = 0;
                col[u] = (int)(v << 4);
                if (rows_per_unit > 1) {
                    lr[u] = (int)(div_magic ? __umulhi(v, div_magic) : v / vec_per_row);
                    col[u] = (int)((v - (uint32_t)lr[u] * vec_per_row) << 4);
                }
                if (v < total && (!BLK || col[u] < a.in_features)) {
                    const int64_t row = (int64_t)a.row0 + lr0 + lr[u];
                    q[u] = ld_stream_u4(a.idx + row * a.ld_idx + col[u]);
                    if (STM) {    // group_size % 16 == 0 and col0 % 16 == 0 on this path: one group per piece
                        const int c = a.col0 + col[u];
                        const int64_t o = row * a.ld_st + (group_shift >= 0 ? c >> group_shift : c / a.group_size) - g_base;
                        s[u] = STM == 1 ? reinterpret_cast<const float*>(a.scales)[o] : __half2float(reinterpret_cast<const __half*>(a.scales)[o]);
                        t[u] = STM == 1 ? reinterpret_cast<const float*>(a.offsets)[o] : __half2float(reinterpret_cast<const __half*>(a.offsets)[o]);
                    }
                }
            }
            if (a.rowptr != nullptr && v0 == first + lane && e0 + lane < e1) {
                sc_col = a.cols[e0 + lane];
                if (a.values != nullptr) sc_val = a.values[e0 + lane];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v0 + 32 * u >= total) break;
                const uint32_t words[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
                uint32_t w[16];       // fp32 bits
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const uint32_t off = __byte_perm(words[j >> 2], lane4, 0x5504u | (uint32_t)((j & 3) << 4));        // code * 256 + lane * 4
                    const float c = *reinterpret_cast<const float*>(lut + off);
                    w[j] = __float_as_uint(STM ? affine_2round(c, s[u], t[u]) : c);
                }
                const int64_t o = out_at<BLK>(a, lr0 + lr[u], col[u]);
                if (BLK && col[u] >= a.in_features) {      // zeros up to the whole step
#pragma unroll
                    for (int j = 0; j < 16; ++j) w[j] = 0u;
                }
                if (OUT_DT == HXQ_F32) {
                    float* dst = reinterpret_cast<float*>(a.out) + o;
                    if (a.wide) {
                        st_global_32(dst, w);
                        st_global_32(dst + 8, w + 8);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(dst)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                    }
                } else {
                    uint32_t pk[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float lo = __uint_as_float(w[2 * j]), hi = __uint_as_float(w[2 * j + 1]);
                        if (OUT_DT == HXQ_BF16) {
                            __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
                            pk[j] = *reinterpret_cast<uint32_t*>(&h);
                        } else {
                            __half2 h = __floats2half2_rn(lo, hi);
                            pk[j] = *reinterpret_cast<uint32_t*>(&h);
                        }
                    }
                    uint16_t* dst = reinterpret_cast<uint16_t*>(a.out) + o;
                    if (a.wide) {
                        st_global_32(dst, pk);
                    } else {
                        reinterpret_cast<uint4*>(dst)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        reinterpret_cast<uint4*>(dst)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                    }
                }
            }
        }
        if (a.rowptr != nullptr) {
            __syncwarp();             // the unit's dense values are written
            const int c_lo = segs > 1 ? (int)first << 4 : 0, c_hi = segs > 1 ? (int)total << 4 : a.in_features;
            if (sc_col >= c_lo && sc_col < c_hi)
                sidecar_entry<BLK>(a, lr0, sc_col, a.values != nullptr ? sc_val : sidecar_value(a, a.row0 + lr0, sc_col, e0 + lane), OUT_DT);
            for (int e = e0 + lane + 32; e < e1; e += 32) {
                const int c = a.cols[e];
                if (c >= c_lo && c < c_hi) sidecar_entry<BLK>(a, lr0, c, sidecar_value(a, a.row0 + lr0, c, e), OUT_DT);
            }
            for (int r = 1; r < nr; ++r) sidecar_row<BLK>(a, lr0 + r, lane, OUT_DT);
        }
    }
}

// Scalar path for ragged / unaligned shapes.
__global__ void __launch_bounds__(256) dequant_scalar_kernel(DequantArgs a, int out_dt) {
    __shared__ float cb_s[256];
    cb_s[threadIdx.x] = a.cb[threadIdx.x];
    __syncthreads();
    const int64_t total = (int64_t)(a.row1 - a.row0) * a.in_features;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int lr = (int)(e / a.in_features);
        const int col = (int)(e - (int64_t)lr * a.in_features);
        const int row = a.row0 + lr;
        float w = weight_at(a, cb_s, row, col, a.idx[(int64_t)row * a.ld_idx + col]);
        store_from_f32(a.out, (int64_t)lr * a.ld_out + col, w, out_dt);
    }
}

// Sidecar of the scalar path: one warp per row.
__global__ void __launch_bounds__(256) dequant_sidecar_kernel(DequantArgs a, int out_dt) {
    const int lr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (a.row0 + lr < a.row1) sidecar_row<false>(a, lr, threadIdx.x & 31, out_dt);
}

template <int OUT_DT, int STM, bool BLK>
static int launch_vec_stm(const DequantArgs& a, cudaStream_t stream) {
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(dequant_vec_kernel<OUT_DT, STM, BLK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVecLutBytes) != cudaSuccess)
            return HXQ_E_DEVICE;
        attr_set[dev] = true;
    }
    const int vec_per_row = a.k_pad >> 4;
    const int rows = a.row1 - a.row0;
    // pieces per unit: 256, fewer (in whole warps) when the matrix would not go round the resident warps twice - a
    // 512 x 3584 one in units of a row ran on 32 SMs
    const int64_t share = (int64_t)rows * vec_per_row / (148 * 2 * (kVecThreads / 32) * 2) / 32 * 32;
    const int pieces = share < 32 ? 32 : (share > kUnitPieces ? kUnitPieces : (int)share);
    const int per_unit = vec_per_row * 2 > pieces ? 1 : pieces / vec_per_row;
    const int segs = per_unit > 1 ? 1 : (vec_per_row + pieces - 1) / pieces;
    const int64_t blocks64 = ((int64_t)((rows + per_unit - 1) / per_unit) * segs + kVecThreads / 32 - 1) / (kVecThreads / 32);
    const int blocks = (int)(blocks64 < 148 * 2 ? blocks64 : 148 * 2);
    int shift = -1;
    if (a.group_size > 0 && (a.group_size & (a.group_size - 1)) == 0)
        for (shift = 0; (1 << shift) < a.group_size; ) ++shift;
    // v / vec_per_row as a multiplication, for units of several rows: v < 256 (exact while v * vec_per_row < 2^32)
    const uint32_t magic = vec_per_row > 1 ? (uint32_t)(((1ull << 32) + vec_per_row - 1) / vec_per_row) : 0u;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kVecThreads);
    cfg.dynamicSmemBytes = kVecLutBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the table is built while the previous kernel drains
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (BLK && !g_weights_on_stream) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, dequant_vec_kernel<OUT_DT, STM, BLK>, a, per_unit, segs, shift, magic) == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}
template <int OUT_DT, bool BLK>
static int launch_vec(const DequantArgs& a, cudaStream_t stream) {
    return a.group_size == 0 ? launch_vec_stm<OUT_DT, 0, BLK>(a, stream)
                             : (a.st_dtype == HXQ_F32 ? launch_vec_stm<OUT_DT, 1, BLK>(a, stream) : launch_vec_stm<OUT_DT, 2, BLK>(a, stream));
}

static DequantArgs dequant_args(const hxq_desc* d, int32_t row0, int32_t row1, void* out, int64_t ld_out) {
    DequantArgs a;
    a.idx = d->indices; a.cb = d->codebook; a.scales = d->scales; a.offsets = d->offsets;
    a.rowptr = d->rowptr; a.cols = d->cols; a.values = nullptr; a.deltas = d->deltas; a.out = out;
    a.ld_idx = d->ld_idx; a.ld_out = ld_out; a.row0 = row0; a.row1 = row1;
    a.in_features = a.k_pad = d->in_features; a.col0 = d->col0; a.group_size = d->group_size;
    a.ld_st = d->ld_st; a.st_dtype = d->st_dtype; a.wide = 0;
    return a;
}

// The dense product's operand: rows [row0, row1) as bf16 in blocked layout, 32-byte aligned, sidecar as
// W^ + delta (what a product adds).  The caller has checked that the fast path takes the descriptor.
int dequant_blocked(const hxq_desc* d, int32_t row0, int32_t row1, __nv_bfloat16* out, cudaStream_t stream) {
    DequantArgs a = dequant_args(d, row0, row1, out, 0);
    a.k_pad = (d->in_features + 63) / 64 * 64;
    a.wide = 1;
    return launch_vec<HXQ_BF16, true>(a, stream);
}

// Rows [row0, row1) to out, sidecar entries carrying the stored values.
static int dequant_rows(const hxq_desc* d, int32_t row0, int32_t row1, void* out, int out_dtype, int64_t ld_out, cudaStream_t stream) {
    DequantArgs a = dequant_args(d, row0, row1, out, ld_out);
    a.values = d->values;
    const int esz = dtype_size(out_dtype);
    const bool vec = (d->in_features % 16 == 0) && (d->ld_idx % 16 == 0) && aligned_to(d->indices, 16) &&
                     aligned_to(out, 16) && ((ld_out * esz) % 16 == 0) &&
                     (d->group_size == 0 || (d->group_size % 16 == 0 && d->col0 % 16 == 0));
    a.wide = aligned_to(out, 32) && (ld_out * esz) % 32 == 0;
    const int64_t rows = row1 - row0;
    if (vec) {
        const int st = out_dtype == HXQ_F32 ? launch_vec<HXQ_F32, false>(a, stream)
                                            : (out_dtype == HXQ_BF16 ? launch_vec<HXQ_BF16, false>(a, stream) : launch_vec<HXQ_F16, false>(a, stream));
        if (st != HXQ_OK) return st;
    } else {
        int64_t total = rows * d->in_features;
        int64_t blocks = (total + 255) / 256;
        if (blocks > 148 * 16) blocks = 148 * 16;
        dequant_scalar_kernel<<<(int)blocks, 256, 0, stream>>>(a, out_dtype);
        if (d->rowptr) {
            if (cudaGetLastError() != cudaSuccess) return HXQ_E_LAUNCH;
            dequant_sidecar_kernel<<<(int)((rows * 32 + 255) / 256), 256, 0, stream>>>(a, out_dtype);
        }
    }
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

}  // namespace hxq

extern "C" int hxq_dequant(const hxq_desc* d, int32_t row0, int32_t row1, void* out, int out_dtype,
                           int64_t ld_out, hxq_stream_t stream_) {
    using namespace hxq;
    int st = validate_desc(d);
    if (st != HXQ_OK) return st;
    if (!out) return HXQ_E_ARG;
    if (!dtype_ok(out_dtype)) return HXQ_E_DTYPE;
    if (row0 < 0 || row1 > d->out_features || row0 > row1) return HXQ_E_SHAPE;
    if (ld_out < d->in_features) return HXQ_E_SHAPE;
    if (d->rowptr && !d->values) return HXQ_E_ARG;
    if (row0 == row1) return HXQ_OK;
    return dequant_rows(d, row0, row1, out, out_dtype, ld_out, reinterpret_cast<cudaStream_t>(stream_));
}

// The encoder's passes over a dense weight: order statistics, nearest-code assignment, outlier
// positions and the per-group affine fit.  All of them stream the weight (4 bytes
// a value) once per pass and do little per value: bound by memory, a weight of up to 126 MB by L2.
//
// The torch operators they replace spent over 100 ms on a 3584 x 3584 weight: kthvalue works a whole
// tensor with one thread block, and the fit made a dozen fp64 copies of the weight.  Here: the two selections 45 us, an
// assignment 29, the outlier passes 22, the fit 48.

#include "hxq_common.cuh"

namespace hxq {
namespace enc {

constexpr int WARP_RUN = 1024;            // values a warp walks in the outlier passes

// Total order of fp32 as unsigned keys; every NaN last, as the sorts of numpy and torch have it.
__device__ __forceinline__ uint32_t key_of(float v) {
    const uint32_t u = __float_as_uint(v);
    if ((u & 0x7fffffffu) > 0x7f800000u) return 0xffffffffu;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) {
    if (k == 0xffffffffu) return __uint_as_float(0x7fc00000u);
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// ---- two order statistics by radix selection, most significant bits first: 11 + 11 + 10 ----------
// Both ranks share the three passes over the data.  A pass counts, in shared memory, the next digit
// of the values that still match a rank's prefix; a one-block kernel then picks the digit.
struct SelectState {
    int64_t rank[2];          // rank left inside the prefix
    uint32_t prefix[2];
};
constexpr int BINS = 2048;

template <int PASS>
__global__ void __launch_bounds__(512) select_count_kernel(const float* __restrict__ v, int64_t n, const SelectState* st,
                                                           unsigned int* __restrict__ hist) {
    constexpr int SETS = PASS == 0 ? 1 : 2;
    __shared__ unsigned int h[SETS * BINS];
    for (int i = threadIdx.x; i < SETS * BINS; i += blockDim.x) h[i] = 0u;
    const uint32_t p0 = PASS == 0 ? 0u : st->prefix[0], p1 = PASS == 0 ? 0u : st->prefix[1];
    __syncthreads();
    auto count = [&](float f) {
        const uint32_t k = key_of(f);
        if (PASS == 0) {
            atomicAdd(&h[k >> 21], 1u);
        } else {
            const uint32_t top = PASS == 1 ? k >> 21 : k >> 10;
            const uint32_t digit = PASS == 1 ? (k >> 10) & 2047u : k & 1023u;
            if (top == p0) atomicAdd(&h[digit], 1u);
            if (top == p1) atomicAdd(&h[BINS + digit], 1u);
        }
    };
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    const bool vec = (reinterpret_cast<uintptr_t>(v) & 15) == 0;
    const int64_t n4 = vec ? n >> 2 : 0;
    for (int64_t i = t; i < n4; i += step) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(v) + i);
        count(f.x); count(f.y); count(f.z); count(f.w);
    }
    for (int64_t i = 4 * n4 + t; i < n; i += step) count(v[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < SETS * BINS; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

// One block of 1024 threads: the digit that holds each rank, and the rank inside it.
template <int PASS>
__global__ void __launch_bounds__(1024) select_pick_kernel(const unsigned int* __restrict__ hist, SelectState* st, float* out) {
    __shared__ unsigned int scan[1024];
    const int t = threadIdx.x;
    for (int w = 0; w < 2; ++w) {
        const unsigned int* h = hist + (PASS == 0 ? 0 : w * BINS);
        const unsigned int a = h[2 * t], b = h[2 * t + 1];
        scan[t] = a + b;
        __syncthreads();
        for (int off = 1; off < 1024; off <<= 1) {
            const unsigned int add = t >= off ? scan[t - off] : 0u;
            __syncthreads();
            scan[t] += add;
            __syncthreads();
        }
        const int64_t below = (int64_t)scan[t] - a - b, rank = st->rank[w];
        __syncthreads();          // every thread has the rank before one of them replaces it
        if (rank >= below && rank < below + a + b) {
            const bool second = rank >= below + a;
            st->rank[w] = rank - below - (second ? a : 0);
            const uint32_t digit = 2 * t + (second ? 1 : 0);
            const uint32_t p = PASS == 0 ? digit : (st->prefix[w] << (PASS == 1 ? 11 : 10)) | digit;
            st->prefix[w] = p;
            if (PASS == 2) out[w] = value_of(p);
        }
        __syncthreads();
    }
}

__global__ void select_init_kernel(SelectState* st, int64_t r0, int64_t r1) {
    st->rank[0] = r0; st->rank[1] = r1;
    st->prefix[0] = st->prefix[1] = 0u;
}

// ---- nearest code ----------------------------------------------------------------------------------
// index = number of midpoints below the value.  A midpoint of two fp32 codes is exact in fp64; the
// largest fp32 not above it separates the same fp32 values, so the search compares fp32.  The 255
// separators are stored breadth first: the nodes of one level of the search are neighbours, so the
// warp's 32 different paths read 32 different banks on the first six levels (in value order they met
// in one or two banks from the third level on).
__global__ void __launch_bounds__(256) assign_kernel(const float* __restrict__ w, int64_t n, const float* __restrict__ cb, int k,
                                                     uint8_t* __restrict__ idx) {
    __shared__ float tree[256];
    {
        const int node = threadIdx.x;
        if (node >= 1) {
            const int level = 31 - __clz(node), pos = node - (1 << level);
            const int i = ((2 * pos + 1) << (7 - level)) - 1;        // separator i is between codes i and i + 1
            float t = __int_as_float(0x7f800000);
            if (i < k - 1) {
                const double mid = ((double)cb[i] + (double)cb[i + 1]) * 0.5;
                t = __double2float_rd(mid);
            }
            tree[node] = t;
        }
    }
    __syncthreads();
    auto code_of = [&](float v) -> uint32_t {
        int node = 1;
#pragma unroll
        for (int l = 0; l < 8; ++l) node = 2 * node + (tree[node] >= v ? 0 : 1);     // (a NaN goes right)
        node -= 256;
        return (uint32_t)(node < k - 1 ? node : k - 1);
    };
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(w) & 15) | (reinterpret_cast<uintptr_t>(idx) & 3)) == 0;
    const int64_t n4 = vec ? n >> 2 : 0;
    for (int64_t i = t; i < n4; i += step) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(w) + i);
        reinterpret_cast<uint32_t*>(idx)[i] = code_of(f.x) | code_of(f.y) << 8 | code_of(f.z) << 16 | code_of(f.w) << 24;
    }
    for (int64_t i = 4 * n4 + t; i < n; i += step) idx[i] = (uint8_t)code_of(w[i]);
}

// ---- outliers: values below thr[0] or above thr[1], positions ascending ---------------------------
// A warp owns WARP_RUN consecutive values.  First its count, then (after a scan of the counts by the
// caller) its positions, if it has any.
__global__ void __launch_bounds__(256) outlier_count_kernel(const float* __restrict__ w, int64_t n, const float* __restrict__ thr,
                                                            int32_t* __restrict__ counts) {
    const int64_t run = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int64_t first = run * WARP_RUN;
    if (first >= n) return;
    const float lo = thr[0], hi = thr[1];
    int c = 0;
#pragma unroll 8
    for (int j = 0; j < WARP_RUN; j += 32) {
        const int64_t i = first + j + lane;
        const float v = i < n ? __ldg(w + i) : lo;
        c += (i < n && (v < lo || v > hi)) ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) counts[run] = c;
}
__global__ void __launch_bounds__(256) outlier_fill_kernel(const float* __restrict__ w, int64_t n, const float* __restrict__ thr,
                                                           const int64_t* __restrict__ ends, int64_t* __restrict__ pos,
                                                           float* __restrict__ vals) {
    const int64_t run = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int64_t first = run * WARP_RUN;
    if (first >= n) return;
    int64_t at = run ? ends[run - 1] : 0;
    if (ends[run] == at) return;
    const float lo = thr[0], hi = thr[1];
    for (int j = 0; j < WARP_RUN; j += 32) {
        const int64_t i = first + j + lane;
        const float v = i < n ? __ldg(w + i) : lo;
        const bool hit = i < n && (v < lo || v > hi);
        const unsigned int m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int64_t o = at + __popc(m & ((1u << lane) - 1u));
            pos[o] = i;
            vals[o] = v;
        }
        at += __popc(m);
    }
}

// ---- per-(row, group) least squares of w on its code's value, excluded positions left out -----------
// Eight lanes per group, four groups per warp (a warp per group spent most of its time in the five exchange
// steps of five fp64 sums: 84 us for 100 K groups of 128, this 48): 16 consecutive values per lane where groups
// and addresses allow 16-byte loads, else every eighth.  fp64 sums; `exclude` ascends, so a group's
// entries are one (mostly empty) run of it.
__global__ void __launch_bounds__(256) fit_kernel(const float* __restrict__ w, const uint8_t* __restrict__ idx,
                                                  const float* __restrict__ cb, int64_t n_groups, int group, int vec,
                                                  const int64_t* __restrict__ exclude, int64_t n_ex,
                                                  float* __restrict__ s_out, float* __restrict__ t_out) {
    __shared__ float cb_s[256];
    cb_s[threadIdx.x] = cb[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, sl = lane & 7;
    const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 3;
    for (int64_t g0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane) >> 3; g0 < n_groups; g0 += step) {
        const int64_t g = g0 + (lane >> 3);
        const bool ok = g < n_groups;           // (lanes of a missing group stay in the exchanges)
        const int64_t first = g * group;
        int64_t e0 = 0, e1 = ok ? n_ex : 0;
        while (e0 < e1) {
            const int64_t m = (e0 + e1) >> 1;
            if (exclude[m] < first) e0 = m + 1; else e1 = m;
        }
        const bool any = ok && e0 < n_ex && exclude[e0] < first + group;
        double n = 0, sc = 0, sw = 0, scc = 0, scw = 0;
        int64_t e = e0;       // this lane's place among the group's entries: its own positions ascend too
        auto add = [&](float wv, uint32_t code, int i) {
            if (any) {
                while (e < n_ex && exclude[e] < first + i) ++e;
                if (e < n_ex && exclude[e] == first + i) return;
            }
            const double v = wv, c = cb_s[code];
            n += 1.0;
            sc += c;
            sw += v;
            scc = __dadd_rn(scc, __dmul_rn(c, c));
            scw = __dadd_rn(scw, __dmul_rn(c, v));
        };
        if (ok && vec) {
            for (int i = 16 * sl; i < group; i += 128) {
                const uint4 q = *reinterpret_cast<const uint4*>(idx + first + i);
                const uint32_t word[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 f = *reinterpret_cast<const float4*>(w + first + i + 4 * j);
                    add(f.x, word[j] & 0xffu, i + 4 * j);
                    add(f.y, (word[j] >> 8) & 0xffu, i + 4 * j + 1);
                    add(f.z, (word[j] >> 16) & 0xffu, i + 4 * j + 2);
                    add(f.w, word[j] >> 24, i + 4 * j + 3);
                }
            }
        } else if (ok) {
            for (int i = sl; i < group; i += 8) add(w[first + i], idx[first + i], i);
        }
        __syncwarp();
#pragma unroll
        for (int off = 4; off; off >>= 1) {
            n += __shfl_xor_sync(0xffffffffu, n, off);
            sc += __shfl_xor_sync(0xffffffffu, sc, off);
            sw += __shfl_xor_sync(0xffffffffu, sw, off);
            scc += __shfl_xor_sync(0xffffffffu, scc, off);
            scw += __shfl_xor_sync(0xffffffffu, scw, off);
        }
        if (ok && sl == 0) {
            // products and differences rounded one by one: a group of one code has a determinant of exactly zero
            const double den = __dsub_rn(__dmul_rn(n, scc), __dmul_rn(sc, sc));
            const double num = __dsub_rn(__dmul_rn(n, scw), __dmul_rn(sc, sw));
            const double s = fabs(den) > 1e-30 ? num / den : 1.0;
            const double t = n > 0 ? __dsub_rn(sw, __dmul_rn(s, sc)) / n : 0.0;
            s_out[g] = (float)s;
            t_out[g] = (float)t;
        }
    }
}

static int blocks_for(int64_t threads, int per_block, int limit) {
    const int64_t b = (threads + per_block - 1) / per_block;
    return (int)(b < 1 ? 1 : (b < limit ? b : limit));
}

}  // namespace enc
}  // namespace hxq

extern "C" size_t hxq_encode_select_workspace_bytes(void) { return sizeof(hxq::enc::SelectState) + 5 * hxq::enc::BINS * sizeof(unsigned int); }

extern "C" int hxq_encode_select2(const float* v, int64_t n, int64_t rank0, int64_t rank1, float* out, void* workspace,
                                  size_t workspace_bytes, hxq_stream_t stream_) {
    using namespace hxq::enc;
    if (!v || !out) return HXQ_E_ARG;
    if (n <= 0 || n > 0xffffffffLL || rank0 < 0 || rank0 >= n || rank1 < 0 || rank1 >= n) return HXQ_E_SHAPE;
    if (!workspace || workspace_bytes < hxq_encode_select_workspace_bytes()) return HXQ_E_WORKSPACE;
    if (!hxq::aligned_to(workspace, 8)) return HXQ_E_ALIGN;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    SelectState* st = reinterpret_cast<SelectState*>(workspace);
    unsigned int* hist = reinterpret_cast<unsigned int*>(st + 1);      // 1, 2 and 2 sets of counters
    if (cudaMemsetAsync(hist, 0, 5 * BINS * sizeof(unsigned int), stream) != cudaSuccess) return HXQ_E_LAUNCH;
    select_init_kernel<<<1, 1, 0, stream>>>(st, rank0, rank1);
    const int blocks = blocks_for((n + 3) / 4, 512, 148 * 4);
    select_count_kernel<0><<<blocks, 512, 0, stream>>>(v, n, st, hist);
    select_pick_kernel<0><<<1, 1024, 0, stream>>>(hist, st, out);
    select_count_kernel<1><<<blocks, 512, 0, stream>>>(v, n, st, hist + BINS);
    select_pick_kernel<1><<<1, 1024, 0, stream>>>(hist + BINS, st, out);
    select_count_kernel<2><<<blocks, 512, 0, stream>>>(v, n, st, hist + 3 * BINS);
    select_pick_kernel<2><<<1, 1024, 0, stream>>>(hist + 3 * BINS, st, out);
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

extern "C" int hxq_encode_assign(const float* w, int64_t n, const float* codebook, int32_t k, uint8_t* indices, hxq_stream_t stream) {
    if (!w || !codebook || !indices) return HXQ_E_ARG;
    if (n <= 0 || k <= 0 || k > 256) return HXQ_E_SHAPE;
    hxq::enc::assign_kernel<<<hxq::enc::blocks_for((n + 3) / 4, 256, 148 * 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        w, n, codebook, k, indices);
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

extern "C" int64_t hxq_encode_outlier_runs(int64_t n) { return n <= 0 ? 0 : (n + hxq::enc::WARP_RUN - 1) / hxq::enc::WARP_RUN; }

extern "C" int hxq_encode_outliers(const float* w, int64_t n, const float* thresholds, int32_t* counts, const int64_t* ends,
                                   int64_t* positions, float* values, hxq_stream_t stream_) {
    using namespace hxq::enc;
    if (!w || !thresholds || (!counts && !(ends && positions && values))) return HXQ_E_ARG;
    const int64_t runs = hxq_encode_outlier_runs(n), blocks = (runs + 7) / 8;
    if (n <= 0 || blocks > 0x7fffffffLL) return HXQ_E_SHAPE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (counts) outlier_count_kernel<<<(int)blocks, 256, 0, stream>>>(w, n, thresholds, counts);
    else outlier_fill_kernel<<<(int)blocks, 256, 0, stream>>>(w, n, thresholds, ends, positions, values);
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

extern "C" int hxq_encode_fit(const float* w, const uint8_t* indices, const float* codebook, int64_t n_groups, int32_t group_size,
                              const int64_t* exclude, int64_t n_exclude, float* scales, float* offsets, hxq_stream_t stream) {
    if (!w || !indices || !codebook || !scales || !offsets || (n_exclude > 0 && !exclude)) return HXQ_E_ARG;
    if (n_groups <= 0 || group_size <= 0 || n_exclude < 0) return HXQ_E_SHAPE;
    const int vec = group_size % 16 == 0 && hxq::aligned_to(w, 16) && hxq::aligned_to(indices, 16);
    hxq::enc::fit_kernel<<<hxq::enc::blocks_for(n_groups * 8, 256, 148 * 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        w, indices, codebook, n_groups, group_size, vec, exclude, n_exclude, scales, offsets);
    return cudaGetLastError() == cudaSuccess ? HXQ_OK : HXQ_E_LAUNCH;
}

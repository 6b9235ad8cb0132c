// Projections of a few rows in single precision (sm_100a), the products of a decode position:
//   out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n])        x [M <= 64, K], w [N, K], all fp32
// and, in the same launch, the columns of a second weight for the same rows (token and boundary heads).
//
// Tensor cores have no fp32 operands, and with so few rows the product is a stream of the weight matrix.
// A warp owns kCols columns and a share of K; its lanes lie along K, 16 bytes each, so that every load is 512
// contiguous bytes of one row, and keep kRows x kCols partial sums that are added over the lanes once, at the
// end, by exchanges that halve the number of sums a lane holds.  The warps of a CTA that share columns split K
// in steps of 128 and add up through shared memory in a fixed order: results do not depend on timing.  No shared
// memory is filled first: a weight row is used by one warp of a CTA, and so is an x segment.
// More rows go in passes of sixteen (or eight) over the same columns: one after the other in a CTA, whose weights come
// from L1 in all but the first, or each on a CTA of its own, whose weights then come from L2.
//
// What bounds it: the passes of a CTA move kRows * K * 4 bytes of x each, from 16 rows on more than its weights (M = 8 B
// rows of the second relation-MLP layer), but what counts there is how many passes are in flight; the heads and the packed
// projection are the weights' stream from DRAM (one row, 768 x 16256: 4.1 of 6.5 TB/s).  us a launch in a graph over weights
// that exceed the L2, cuBLAS (with its split-K
// reduction) -> here, and the error against 64 bits: 8 x 3072 x 768 23.6 -> 5.7 (2.3e-7 -> 1.1e-7), 32 x 2048 x 512
// 18.6 -> 6.3 (3.2e-7 -> 1.0e-7), 64 x 3072 x 768 33.2 -> 19.8, 4 x 512 x 256 4.3 -> 2.3, 2 x 512 x 3072 5.7 -> 2.8,
// 1 x 512 x 16256 17.6 -> 8.4, 8 x 768 x 16256 27.8 -> 22.8.
// The first step's weights are requested before the dependency wait: parameters, which no kernel of the step writes.
//
// Stands where the reference calls F.linear on one position's rows: src/relation_lm/inference/packed_cache.py:52-57,
// the second layer of src/relation_lm/models/stacked_relation.py:65-182 and the heads of relation_lm.py:121-124.

#include "rlm_common.cuh"

namespace rlm {
namespace {

constexpr int kFewThreads = 256, kFewWarps = kFewThreads / 32;
constexpr int kFewStep = 128;                   // k-values of one step of a warp

struct FewRowsArgs {
    const float* x;
    int x_stride;
    const float *w0, *w1;                       // w1, bias1, out1: the second weight's
    const float *bias0, *bias1;
    float *out0, *out1;
    int n0, n1;
    int rows, k;
    int k_parts;                                // warps that share columns
};

// kRows rows at a time, kCols columns per warp.  Fewer rows leave registers for more CTAs on an SM, whose loads are what
// a stream needs (one row, 512 x 16256: 11.7 us with two CTAs, 8.4 with four).  Under those caps <4, *> and <2, 4> spill
// 4 to 20 bytes.
// kApart: a pass of kRows rows per CTA (x; y: the columns), else a CTA makes all passes over its columns (x).
template <int kRows, int kCols, bool kApart>
__global__ void __launch_bounds__(kFewThreads, kRows <= 2 ? 4 : kRows <= 4 ? 3 : 2) few_rows_projection_kernel(const FewRowsArgs a) {
    constexpr int kSums = kRows * kCols;
    __shared__ float part_s[kFewWarps][kSums];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = kFewWarps / a.k_parts, part = warp % a.k_parts, group = warp / a.k_parts;
    const int tile = (kApart ? blockIdx.y : blockIdx.x) * groups * kCols, n_all = a.n0 + a.n1;
    const int steps = (a.k + kFewStep - 1) / kFewStep;

    const float* wrow[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) {           // columns beyond the last repeat it (and are not stored)
        const int col = min(tile + group * kCols + c, n_all - 1);
        wrow[c] = (col < a.n0 ? a.w0 : a.w1) + static_cast<size_t>(col < a.n0 ? col : col - a.n0) * a.k;
    }
    const auto load = [&](const float* row, int k) {
        return k < a.k ? *reinterpret_cast<const float4*>(row + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    float4 first[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) first[c] = load(wrow[c], kFewStep * part + 4 * lane);
    griddep_sync();

#pragma unroll 1
    for (int m0 = kApart ? blockIdx.x * kRows : 0; m0 < a.rows; m0 += kApart ? a.rows : kRows) {
        int xrow[kRows];                        // rows beyond the last repeat it (and are not stored)
#pragma unroll
        for (int m = 0; m < kRows; ++m) xrow[m] = min(m0 + m, a.rows - 1) * a.x_stride;
        float sum[kSums];
#pragma unroll
        for (int i = 0; i < kSums; ++i) sum[i] = 0.0f;
        const auto step = [&](int k, const float4 (&w)[kCols]) {
            constexpr int kAtOnce = kRows < 8 ? kRows : 8;
#pragma unroll
            for (int m8 = 0; m8 < kRows; m8 += kAtOnce) {
                float4 xv[kAtOnce];
#pragma unroll
                for (int m = 0; m < kAtOnce; ++m) xv[m] = load(a.x + xrow[m8 + m], k);
#pragma unroll
                for (int m = 0; m < kAtOnce; ++m)
#pragma unroll
                    for (int c = 0; c < kCols; ++c) {
                        float& s = sum[(m8 + m) * kCols + c];
                        s = fmaf(xv[m].x, w[c].x, s);
                        s = fmaf(xv[m].y, w[c].y, s);
                        s = fmaf(xv[m].z, w[c].z, s);
                        s = fmaf(xv[m].w, w[c].w, s);
                    }
            }
        };
        step(kFewStep * part + 4 * lane, first);
#pragma unroll (kRows <= 8 ? 2 : 1)
        for (int i = part + a.k_parts; i < steps; i += a.k_parts) {
            const int k = kFewStep * i + 4 * lane;
            float4 w[kCols];
#pragma unroll
            for (int c = 0; c < kCols; ++c) w[c] = load(wrow[c], k);
            step(k, w);
        }
        // over the lanes: the lanes of either half take half of the sums, until each has one (or shares it)
        int held = 0;
        {
            int n = kSums;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                if (n > 1) {
                    n >>= 1;
                    const bool upper = (lane & o) != 0;
                    held += upper ? n : 0;
#pragma unroll
                    for (int i = 0; i < kSums / 2; ++i)
                        if (i < n) {
                            const float send = upper ? sum[i] : sum[i + n], keep = upper ? sum[i + n] : sum[i];
                            sum[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                } else {
                    sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
                }
            }
        }
        part_s[warp][held] = sum[0];            // lanes that share a sum store the same value
        if (kSums > 32) part_s[warp][held + 1] = sum[kSums > 32 ? 1 : 0];
        __syncthreads();
        for (int at = threadIdx.x; at < groups * kSums; at += kFewThreads) {
            const int g = at / kSums, i = at % kSums, m = m0 + i / kCols, col = tile + g * kCols + i % kCols;
            float v = 0.0f;
            for (int p = 0; p < a.k_parts; ++p) v += part_s[g * a.k_parts + p][i];
            if (m < a.rows && col < n_all) {
                const bool second = col >= a.n0;
                const int column = second ? col - a.n0 : col;
                const float* bias = second ? a.bias1 : a.bias0;
                if (bias) v += bias[column];
                (second ? a.out1 : a.out0)[static_cast<size_t>(m) * (second ? a.n1 : a.n0) + column] = v;
            }
        }
        __syncthreads();
    }
}

template <int kCols>
int few_rows_tiles(const FewRowsArgs& a) {
    const int cols = kFewWarps / a.k_parts * kCols;
    return (a.n0 + a.n1 + cols - 1) / cols;
}

template <int kRows, int kCols>
int launch_few_rows(const FewRowsArgs& a, void* stream) {
    // Passes over rows on CTAs of their own where that makes fewer waves (two CTAs an SM) than a CTA would make passes: a pass
    // is a few dependent loads long, not a stream; where the columns fill the SMs, further passes find their weights in L1.
    // us: 32 x 1024 x 256 3.8 -> 3.3, 32 x 2304 x 576 10.5 -> 7.6, 64 x 2304 x 576 17.6 -> 13.6, 48 x 3072 x 768 19.6 -> 14.6;
    // 32 x 1536 x 768 9.1 -> 9.8 and 64 x 512 x 2304 11.5 -> 12.9, as many waves as passes, stay in one CTA, except where the
    // second wave is at most half full and its passes are long and even: 32 x 2048 x 768 10.3 -> 9.8, 24 x 3072 x 768
    // 13.7 -> 12.4 (but 32 x 2304 x 768 12.6 -> 13.2).  The sums and their order are the same.
    const int tiles = few_rows_tiles<kCols>(a), passes = (a.rows + kRows - 1) / kRows, at_once = 2 * sm_count();
    const bool fewer = (tiles * static_cast<int64_t>(passes) + at_once - 1) / at_once < passes;
    const bool even = 2 * tiles * static_cast<int64_t>(passes) <= 3 * at_once && a.k >= 16 * kFewStep && a.k % (a.k_parts * kFewStep) == 0;
    const bool apart = passes > 1 && tiles <= at_once && (fewer || even);
    if (apart) launch_kernel(few_rows_projection_kernel<kRows, kCols, (kRows >= 8)>, dim3(passes, tiles), dim3(kFewThreads), 0, stream, a);
    else launch_kernel(few_rows_projection_kernel<kRows, kCols, false>, dim3(tiles), dim3(kFewThreads), 0, stream, a);
    count_launch();
    return check_launch("few_rows_projection_kernel");
}

template <int kCols>
int dispatch_few_rows(const FewRowsArgs& a, void* stream) {
    if (a.rows == 1) return launch_few_rows<1, kCols>(a, stream);
    if (a.rows == 2) return launch_few_rows<2, kCols>(a, stream);
    if (a.rows <= 4) return launch_few_rows<4, kCols>(a, stream);
    // Eight rows a pass where all passes then run at once and are long enough to gain by it (us: 16 x 2048 x 512 5.2 -> 4.7,
    // 16 x 2304 x 576 6.8 -> 5.6; 9 x 1024 x 256 2.4 -> 2.55).
    const bool eight = a.rows <= 8 || (a.k >= 16 * kFewStep && few_rows_tiles<kCols>(a) * static_cast<int64_t>((a.rows + 7) / 8) <= 2 * sm_count());
    return eight ? launch_few_rows<8, kCols>(a, stream) : launch_few_rows<16, kCols>(a, stream);
}

}  // namespace
}  // namespace rlm

extern "C" int rlm_few_rows_projection(const float* x, int64_t x_row_stride, const float* weight, const float* bias, float* out,
                                       const float* weight2, const float* bias2, float* out2, int rows, int d_in, int n_out,
                                       int n_out2, void* stream) {
    using namespace rlm;
    if (rows == 0 || n_out + n_out2 == 0) return RLM_OK;
    if (!x || (n_out > 0 && (!weight || !out)) || (n_out2 > 0 && (!weight2 || !out2))) {
        set_error("few_rows_projection: NULL pointer");
        return RLM_ERR_NULL;
    }
    if (rows < 0 || rows > 64 || n_out < 0 || n_out2 < 0 || x_row_stride > 0x1000000 || d_in < 4 || d_in % 4 != 0 || x_row_stride < d_in || x_row_stride % 4 != 0 ||
        static_cast<int64_t>(n_out) + n_out2 > 0x7fffffff - 1024) {
        set_error("few_rows_projection: at most 64 rows, width and row stride multiples of 4");
        return RLM_ERR_SHAPE;
    }
    if (!aligned16(x) || !aligned16(weight) || !aligned16(weight2)) {
        set_error("few_rows_projection: x and the weights must be 16-byte aligned");
        return RLM_ERR_ALIGN;
    }
    FewRowsArgs a{};
    a.x = x; a.x_stride = static_cast<int>(x_row_stride); a.rows = rows; a.k = d_in;
    a.w0 = weight; a.w1 = weight2; a.bias0 = bias; a.bias1 = bias2; a.out0 = out; a.out1 = out2;
    a.n0 = n_out; a.n1 = n_out2;
    // as many warps on a column as there are steps for them; two columns a warp where four leave half of the SMs without a CTA
    const int steps = (d_in + kFewStep - 1) / kFewStep;
    a.k_parts = steps >= 8 ? 8 : steps >= 4 ? 4 : steps >= 2 ? 2 : 1;
    const int groups = (n_out + n_out2 + 3) / 4 / (kFewWarps / a.k_parts);
    return groups >= sm_count() / 2 ? dispatch_few_rows<4>(a, stream) : dispatch_few_rows<2>(a, stream);
}

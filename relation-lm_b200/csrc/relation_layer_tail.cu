// The whole relation tail of one layer in one launch, for decode batches of a few sequences
// (sm_100a): gathers, product term of the first relation-MLP layer, GELU, second relation-MLP
// layer, per-partner LayerNorm, active-K softmax, weighted sum, residual update, the next
// LayerNorm and (optionally) the next layer's query-side projection.  The relation hidden
// states [pairs, H] never leave the chip and no vendor GEMM is called.
//
//   hidden[b,k,:] = gelu(W_m (o[a_b] * o[p_bk]) + E[a_b, 0:H] + E[p_bk, H:2H])     (16-bit, on chip)
//   raw[b,k,:]    = W_2 hidden[b,k,:] + b_2                                        (fp32, on chip)
//   context[b]    = sum_k w_bk LayerNorm(raw[b,k,:]),  w = softmax over the active partner slots
//   residual[b]  += mix * context[b];  normalized[b] = LayerNorm'(residual[b])
//   query[b]      = W_q normalized[b]                                              (optional)
//
// Geometry (d <= 512, few pairs).  A thread-block cluster of C = H / 128 CTAs serves up to 64 (sequence, partner)
// pairs; CTA c owns hidden columns [128 c, 128 c + 128).  Its weight slices — W_m[128 c .., :]
// (128 x R) and W_2[:, 128 c ..] (d x 128) — are requested by TMA before the dependency wait and
// stay resident in shared memory.  After the selector's indices arrive every CTA gathers the
// operand rows (multiplied from registers into the swizzled B tile) and its 128 columns of the two
// expanded-cache terms, runs the product GEMM with the hidden columns on the TMEM lanes
// (tcgen05.mma, pairs on the TMEM columns), applies GELU and writes its hidden slice as the
// K-major B tile of the second GEMM, whose A operand is the resident W_2 slice: a split-K GEMM
// over the cluster, each CTA holding a partial raw^T [d, pairs] in TMEM.
//
// Launches of more than 16 pairs a cluster (d >= 256): the partial sums, C x d x pairs floats through distributed shared
// memory at some 15 bytes a cycle and CTA, become what takes the time (64 pairs: waited for during 8 300 of 32 000 cycles,
// sharing 5 800 of 28 600; 32 pairs 5 300 of 22 500, 3 600 of 20 300).  There
// neighbouring CTAs exchange their 16-bit hidden slices and divide the output rows: each has half of the rows over both
// slices, the partial sums are half as many, and the other's slice travels while the own one is multiplied.
//
// d = 768 (kWide): 16 CTAs of 192 hidden columns (two overlapping tiles of the product GEMM) and 48 output columns, always
// sharing; a CTA's part of W_2, 288 KB, does not fit beside the rest and goes through a ring of six to nine tiles of
// 16 KB, three warps issuing a tile of output rows each and a fourth refilling.  The products of the operand rows keep all
// their bits here (a second tile for what rounding to 16 bits takes off), because the separate kernels that this form
// replaces keep them in fp32: residual rows are 1.61e-4 off 64 bits (bf16, 28 x 8 pairs, root mean square), 2.09e-4 without,
// 2.27e-4 from the separate kernels, for 1 us a layer of 8 sequences.  us a step of 12 layers, context 1024, in a graph,
// five launches a layer -> here: batch 1 303 -> 250, batch 8 341 -> 269, batch 16 407 -> 324, batch 28 483 -> 400.
//
// us a step of 6 layers of d 512 before sharing, the gathers through registers, two issuing warps and the statistics in
// messages of two pairs -> with them: batch 1 84.0 -> 81.9, 5 98.4 -> 94.3, 8 97.5 -> 94.3, 16 128.5 -> 122.5,
// 32 167.6 -> 157.3, 48 174.1 -> 164.0.
//
// What bounds the launch is a chain of some twenty dependent phases, so the CTAs hand their results on by pushing
// them into the receiver's shared memory with stores that count towards a barrier of the receiver (st.async), and a
// receiver waits for exactly what it needs: no cluster-wide barrier lies in the chain and no remote load.  Three
// exchanges: the partial sums go from the accumulators straight to the CTA that owns the output row (d / C rows
// each, summed in rank order: deterministic); (mean, M2) of a CTA's 32 columns per pair to every CTA (Chan's
// parallel variance); the updated residual columns to every CTA, which then normalises whole rows for its share of
// the query projection.  Cluster barriers remain off the chain: one split in two halves around the second GEMM (the
// weight slice whose place receives the partial sums has been consumed everywhere), one around the projection (no
// CTA leaves while another may still push to it).  With four cluster barriers, partial sums dumped and pulled and
// normalised rows stored value by value, a step of the 6-layer model took 150 us at batch 1, now 139 us.
//
// Semantics follow src/relation_lm/kernels/relation_reduce.py:72-146 and 360-417 of the
// reference project with the cuBLAS second layer of benchmarks/benchmark_relation_reduce.py:55-64
// in between, and `hidden + sigmoid(mix) * context` of models/stacked_relation.py:124.
// Every wait is bounded; on expiry the kernel sets RLM_DEV_TIMEOUT, still pushes what it owes and passes every cluster
// barrier (so no CTA waits for a peer that left), frees its TMEM and returns.

#include "relation_layer_tail_body.cuh"

namespace rlm {
namespace {

template <bool kBf16, bool kAligned, bool kWide, bool kMany>
__global__ void __launch_bounds__(kLtThreads, 1) relation_layer_tail_kernel(
    const __grid_constant__ CUtensorMap map_wm, const __grid_constant__ CUtensorMap map_w2,
    const LayerTailArgs a) {
    extern __shared__ __align__(1024) unsigned char lt_smem_raw[];
    layer_tail_body<kBf16, kAligned, kWide, kMany>(map_wm, map_w2, a, lt_smem_raw, NoStage{});
}

using TailKernel = void (*)(const CUtensorMap, const CUtensorMap, const LayerTailArgs);

template <bool kWide, bool kMany>
TailKernel tail_kernel(bool bf16, bool aligned) {
    return aligned ? (bf16 ? relation_layer_tail_kernel<true, true, kWide, kMany> : relation_layer_tail_kernel<false, true, kWide, kMany>)
                   : (bf16 ? relation_layer_tail_kernel<true, false, kWide, kMany> : relation_layer_tail_kernel<false, false, kWide, kMany>);
}
TailKernel tail_kernel(bool bf16, bool aligned, bool wide, bool many) {
    return wide ? (many ? tail_kernel<true, true>(bf16, aligned) : tail_kernel<true, false>(bf16, aligned))
                : (many ? tail_kernel<false, true>(bf16, aligned) : tail_kernel<false, false>(bf16, aligned));
}

// A few sequences per cluster: up to four clusters share the work of a small batch (each
// streams the layer's weights from L2 once), more clusters only for batches beyond 32.
int tail_seqs_per_cluster(int n_seq, int k_out) {
    const int most = kLtMaxPairs / k_out < kLtMaxSeq ? kLtMaxPairs / k_out : kLtMaxSeq;
    return (n_seq + 3) / 4 < most ? (n_seq + 3) / 4 : most;
}

int tail_supported(bool wide, int n_seq, int k_out, int relation_dim, int hidden_dim, int d_model, int n_query, int dtype) {
    LayerTailArgs a{};
    a.n_seq = n_seq; a.k_out = k_out; a.max_t = 1; a.rdim = relation_dim; a.hdim = hidden_dim; a.d = d_model;
    a.n_query = n_query; a.dtype = dtype;
    a.query_weight = n_query > 0 ? &a : nullptr;      // only tested for NULL
    a.query = n_query > 0 ? &a : nullptr;
    if (lt_validate(a, wide) != RLM_OK) return 0;
    const int cluster = lt_cluster(d_model);
    auto kernel = tail_kernel(dtype == RLM_BF16, true, wide, lt_many(tail_seqs_per_cluster(n_seq, k_out), k_out));
    if (lt_prepare(reinterpret_cast<const void*>(kernel), cluster) != RLM_OK) return 0;
    // one cluster of this size, with this much shared memory per CTA, must fit the device
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(cluster, 1, 1);
    config.blockDim = dim3(kLtThreads, 1, 1);
    config.dynamicSmemBytes = lt_smem_bytes(relation_dim, d_model, n_query / cluster);
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = cluster;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters > 0 ? 1 : 0;
}

int launch_tail(bool wide, const void* expanded_cache, const void* operand_cache, const int32_t* anchor_index,
    const int32_t* partner_index, const float* partner_scores, const void* product_weight,
    const void* second_weight, const void* second_bias, const float* norm_weight, const float* norm_bias,
    const int64_t* position, float norm_eps, float* residual, const float* mix,
    const float* next_norm_weight, const float* next_norm_bias, float next_norm_eps, void* normalized,
    const void* query_weight, void* query, int n_seq, int k_out, int max_t, int relation_dim,
    int hidden_dim, int d_model, int n_query, int dtype, int32_t* status, void* stream) {
    if (n_seq == 0) return RLM_OK;
    if (!expanded_cache || !operand_cache || !anchor_index || !partner_index || !partner_scores ||
        !product_weight || !second_weight || !second_bias || !norm_weight || !norm_bias || !position ||
        !residual || !mix || !next_norm_weight || !next_norm_bias || !normalized) {
        set_error("relation_layer_tail: NULL pointer");
        return RLM_ERR_NULL;
    }
    LayerTailArgs a{};
    a.expanded_cache = expanded_cache; a.operand_cache = operand_cache; a.anchor_index = anchor_index;
    a.partner_index = partner_index; a.partner_scores = partner_scores; a.second_bias = second_bias;
    a.norm_w = norm_weight; a.norm_b = norm_bias; a.position = position; a.residual = residual; a.mix = mix;
    a.next_w = next_norm_weight; a.next_b = next_norm_bias; a.normalized = normalized;
    a.query_weight = query_weight; a.query = query; a.status = status; a.eps = norm_eps; a.next_eps = next_norm_eps;
    a.n_seq = n_seq; a.k_out = k_out; a.max_t = max_t; a.rdim = relation_dim; a.hdim = hidden_dim; a.d = d_model;
    a.n_query = query_weight ? n_query : 0; a.dtype = dtype;
    int rc = lt_validate(a, wide);
    if (rc != RLM_OK) return rc;
    if (!aligned16(expanded_cache) || !aligned16(operand_cache) || !aligned16(product_weight) ||
        !aligned16(second_weight) || (query_weight && !aligned16(query_weight))) {
        set_error("relation_layer_tail: caches and weights must be 16-byte aligned");
        return RLM_ERR_ALIGN;
    }
    a.cluster = lt_cluster(d_model);
    a.seqs_per_cluster = tail_seqs_per_cluster(n_seq, k_out);
    const int clusters = (n_seq + a.seqs_per_cluster - 1) / a.seqs_per_cluster;
    CUtensorMap mwm, mw2;
    if (!make_map(&mwm, product_weight, hidden_dim, relation_dim, relation_dim, lt_hidden(d_model), dtype) ||
        !make_map(&mw2, second_weight, d_model, hidden_dim, hidden_dim, kBM, dtype)) {
        set_error("relation_layer_tail: cuTensorMapEncodeTiled failed");
        return RLM_ERR_LAUNCH;
    }
    auto kernel = tail_kernel(dtype == RLM_BF16, lt_aligned(a), wide, lt_many(a.seqs_per_cluster, k_out));
    rc = lt_prepare(reinterpret_cast<const void*>(kernel), a.cluster);
    if (rc != RLM_OK) return rc;
    const size_t smem_bytes = lt_smem_bytes(relation_dim, d_model, a.n_query / a.cluster);
    launch_kernel_cluster(kernel, dim3(a.cluster, clusters), dim3(kLtThreads),
                          static_cast<unsigned>(a.cluster), smem_bytes, stream, mwm, mw2, a);
    count_launch();
    return check_launch("relation_layer_tail_kernel");
}

}  // namespace
}  // namespace rlm

extern "C" int rlm_relation_layer_tail_supported(int n_seq, int k_out, int relation_dim, int hidden_dim, int d_model, int n_query,
                                                 int dtype) {
    return rlm::tail_supported(false, n_seq, k_out, relation_dim, hidden_dim, d_model, n_query, dtype);
}

extern "C" int rlm_relation_layer_tail_wide_supported(int n_seq, int k_out, int relation_dim, int hidden_dim, int d_model,
                                                      int n_query, int dtype) {
    return rlm::tail_supported(true, n_seq, k_out, relation_dim, hidden_dim, d_model, n_query, dtype);
}

extern "C" int rlm_relation_layer_tail(

    const void* expanded_cache, const void* operand_cache, const int32_t* anchor_index,
    const int32_t* partner_index, const float* partner_scores, const void* product_weight,
    const void* second_weight, const void* second_bias, const float* norm_weight, const float* norm_bias,
    const int64_t* position, float norm_eps, float* residual, const float* mix,
    const float* next_norm_weight, const float* next_norm_bias, float next_norm_eps, void* normalized,
    const void* query_weight, void* query, int n_seq, int k_out, int max_t, int relation_dim,
    int hidden_dim, int d_model, int n_query, int dtype, int32_t* status, void* stream) {
    return rlm::launch_tail(false, expanded_cache, operand_cache, anchor_index, partner_index, partner_scores, product_weight, second_weight, second_bias, norm_weight, norm_bias, position, norm_eps, residual, mix, next_norm_weight, next_norm_bias, next_norm_eps, normalized, query_weight, query, n_seq, k_out, max_t, relation_dim, hidden_dim, d_model, n_query, dtype, status, stream);
}

extern "C" int rlm_relation_layer_tail_wide(

    const void* expanded_cache, const void* operand_cache, const int32_t* anchor_index,
    const int32_t* partner_index, const float* partner_scores, const void* product_weight,
    const void* second_weight, const void* second_bias, const float* norm_weight, const float* norm_bias,
    const int64_t* position, float norm_eps, float* residual, const float* mix,
    const float* next_norm_weight, const float* next_norm_bias, float next_norm_eps, void* normalized,
    const void* query_weight, void* query, int n_seq, int k_out, int max_t, int relation_dim,
    int hidden_dim, int d_model, int n_query, int dtype, int32_t* status, void* stream) {
    return rlm::launch_tail(true, expanded_cache, operand_cache, anchor_index, partner_index, partner_scores, product_weight, second_weight, second_bias, norm_weight, norm_bias, position, norm_eps, residual, mix, next_norm_weight, next_norm_bias, next_norm_eps, normalized, query_weight, query, n_seq, k_out, max_t, relation_dim, hidden_dim, d_model, n_query, dtype, status, stream);
}

extern "C" int rlm_selftest_layer_tail_plan(int pairs, int n_seq, int relation_dim, int d_model, int n_query, int64_t* ranges) {
    using namespace rlm;
    if (!ranges) { set_error("selftest_layer_tail_plan: result required"); return RLM_ERR_NULL; }
    const int cluster = d_model < kBM ? 1 : lt_cluster(d_model), pairs_pad = pairs <= 16 ? 16 : (pairs <= 32 ? 32 : 64);
    if (pairs < 1 || pairs > kLtMaxPairs || n_seq < 1 || n_seq > kLtMaxSeq || d_model % kBM != 0 || d_model < kBM || cluster > 16 ||
        (lt_wide(d_model) && d_model != 768) || relation_dim % kBK != 0 || n_query % cluster != 0) {
        set_error("selftest_layer_tail_plan: sizes outside the kernel's range");
        return RLM_ERR_SHAPE;
    }
    const int nq_own = n_query / cluster;
    const LtPlan p = lt_plan(relation_dim, d_model, pairs > 16, pairs_pad, nq_own);
    const int64_t begin[] = {p.own_y, p.rows, p.rows_in, p.term_p, p.wq, 0};
    const int64_t bytes[] = {pairs * (lt_owned(d_model) + 1) * 4, n_seq * d_model * 2, n_seq * d_model * 4, cluster * pairs_pad * 8,
                             nq_own * (2 * d_model + 256), p.total};
    for (int i = 0; i < 6; ++i) { ranges[2 * i] = begin[i]; ranges[2 * i + 1] = begin[i] + bytes[i]; }
    return RLM_OK;
}

// Body of the relation layer tail (see relation_layer_tail.cu for the description) and its host-side
// helpers, shared by the standalone kernel and by the whole-layer kernel that runs the selector
// in front of it (relation_select.cu).
#pragma once

#include <mutex>

#include "rlm_tcgen05.cuh"

namespace rlm {
namespace {

constexpr int kLtThreads = 256;
constexpr int kLtHC = 128;            // hidden columns per CTA
constexpr int kLtMaxPairs = 64;       // (sequence, partner) pairs per cluster
constexpr int kLtMaxSeq = 8;          // sequences per cluster
constexpr int kLtOwn = 32;            // output columns a CTA owns after the reduce-scatter (d / C)
constexpr int kLtOwnStride = 33;      // padded row of the owned raw values (floats)
constexpr uint32_t kLtTermStride = kLtHC * 2 + 16;   // padded row of the staged expanded-cache terms

struct LayerTailArgs {
    const void* expanded_cache;      // [B, T, 2H]
    const void* operand_cache;       // [B, T, R]
    const int32_t* anchor_index;     // [B]
    const int32_t* partner_index;    // [B, K]
    const float* partner_scores;     // [B, K]
    const void* second_bias;         // [d]
    const float* norm_w;             // [d] relation LayerNorm
    const float* norm_b;
    const int64_t* position;
    float* residual;                 // [B, d] in/out
    const float* mix;
    const float* next_w;             // [d] next LayerNorm
    const float* next_b;
    void* normalized;                // [B, d] 16-bit out
    const void* query_weight;        // [NQ, d] or NULL
    void* query;                     // [B, NQ] 16-bit out
    int32_t* status;
    float eps, next_eps;
    int n_seq, k_out, max_t, rdim, hdim, d, n_query, dtype;
    int seqs_per_cluster, cluster;   // cluster = H / 128
};

// Shared-memory plan (byte offsets from the 1024-aligned dynamic base).
struct LtPlan {
    uint32_t wm, w2, p, hid, term_p, term_a, op_a, wq, total;
    uint32_t own_y, rows;                // later uses of p and w2: see lt_plan
};

// The partial sums that a CTA receives, [sender][four pairs][owned column][pair] of 512 d pairs / 128 bytes in all,
// take the place of a consumed weight slice: W_m's for 16 pairs, W_2's for more (the W_q slice then waits for W_m's).
// nq_own: rows of the query-projection weight per CTA.
__host__ __device__ inline LtPlan lt_plan(int rdim, int d, int pairs_pad, int nq_own) {
    LtPlan p;
    uint32_t off = 0;
    const uint32_t received = 4u * static_cast<uint32_t>(d) * pairs_pad;
    p.wm = off;     off += static_cast<uint32_t>(rdim / kBK) * kBM * 128u;           // W_m slice
    if (pairs_pad == 16 && off < received) off = received;
    p.w2 = off;     off += static_cast<uint32_t>(d / kBM) * 2u * kBM * 128u;         // W_2 slice
    p.p = off;      off += static_cast<uint32_t>(rdim / kBK) * pairs_pad * 128u;     // product tile; later the normalised pairs
    if (off - p.p < pairs_pad * kLtOwnStride * 4u) off = p.p + pairs_pad * kLtOwnStride * 4u;
    off = (off + 1023u) & ~1023u;
    p.hid = off;    off += 2u * pairs_pad * 128u;                                    // hidden tile; later the residual rows
    if (off - p.hid < static_cast<uint32_t>(kLtMaxSeq) * d * 4u) off = p.hid + kLtMaxSeq * d * 4u;
    p.term_p = off; off += pairs_pad * kLtTermStride;
    p.term_a = off; off += kLtMaxSeq * kLtTermStride;
    p.op_a = off;   off += kLtMaxSeq * static_cast<uint32_t>(rdim) * 2u;
    p.wq = p.wm;
    if (pairs_pad == 16) { p.wq = off; off += static_cast<uint32_t>(nq_own) * (2u * d + 256u); }
    p.total = off;
    // The last LayerNorm's rows take W_2's place, not the normalised pairs': a warp may write its rows while another
    // of its CTA still sums its pairs (the barrier between them counts what this CTA is sent, and only one warp a
    // sequence sends to it).  W_2's place is free in every warp by then: the statistics that a CTA waits for include
    // its own, and those follow its second GEMM and its reads of the partial sums.
    p.own_y = p.p;
    p.rows = p.w2;
    return p;
}

// Dynamic shared memory of a launch, whatever its pairs per cluster.
inline uint32_t lt_smem_bytes(int rdim, int d, int nq_own) {
    uint32_t most = 0;
    for (int pairs = 16; pairs <= kLtMaxPairs; pairs *= 2) {
        const uint32_t total = lt_plan(rdim, d, pairs, nq_own).total;
        if (total > most) most = total;
    }
    return most + 1024;
}

// Dynamic shared memory of a whole-layer launch, whose stage needs `stage` bytes behind the weight slices.
inline uint32_t lt_smem_bytes_with_stage(int rdim, int d, int nq_own, int stage) {
    uint32_t most = lt_smem_bytes(rdim, d, nq_own);
    for (int pairs = 16; pairs <= kLtMaxPairs; pairs *= 2) {
        const uint32_t total = lt_plan(rdim, d, pairs, nq_own).p + static_cast<uint32_t>(stage) + 1024u;
        if (total > most) most = total;
    }
    return most;
}

__device__ __forceinline__ uint32_t lt_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void lt_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of `local_addr` (a shared-memory address of this CTA) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t lt_peer(uint32_t local_addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    return remote;
}
// Relaxed: no data travels with these barriers (a consumed tile's place is free; nothing more will be pushed), and a
// release would wait a thousand cycles for the warp's earlier stores and copies.
__device__ __forceinline__ void lt_cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void lt_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Stores into another CTA's shared memory that count towards a barrier of that CTA (both addresses from lt_peer).
__device__ __forceinline__ void lt_push16(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void lt_push8(uint32_t addr, uint32_t bar, float x, float y) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
                 ::"r"(addr), "r"(__float_as_uint(x)), "r"(__float_as_uint(y)), "r"(bar) : "memory");
}
__device__ __forceinline__ void lt_push4(uint32_t addr, uint32_t bar, float x) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(addr), "r"(__float_as_uint(x)), "r"(bar) : "memory");
}

// Mean and sum of squared deviations of x[j] over the warp's 32 lanes, for j = lane / 8: equal halves are merged level
// by level (Chan's parallel variance), both values in the same five exchanges.
__device__ __forceinline__ float2 lt_moments4(const float (&x)[4]) {
    const bool hi = threadIdx.x & 16, mid = threadIdx.x & 8;
    float m[2], v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float mine = hi ? x[2 + j] : x[j], other = __shfl_xor_sync(0xffffffffu, hi ? x[j] : x[2 + j], 16), d = mine - other;
        m[j] = 0.5f * (mine + other);
        v[j] = 0.5f * d * d;
    }
    float mean = mid ? m[1] : m[0], m2 = mid ? v[1] : v[0], count = 2.0f;
    float give_mean = mid ? m[0] : m[1], give_m2 = mid ? v[0] : v[1];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, give_mean, o), other2 = __shfl_xor_sync(0xffffffffu, give_m2, o);
        const float d = mean - other;
        m2 = fmaf(d * d, 0.5f * count, m2 + other2);
        mean = 0.5f * (mean + other);
        count += count;
        give_mean = mean;
        give_m2 = m2;
    }
    return make_float2(mean, m2);
}

__device__ __forceinline__ void lt_tmem_ld4(uint32_t addr, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}

template <bool kAligned>
__device__ __forceinline__ float4 lt_load4(const float* p) {
    return kAligned ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

__device__ __forceinline__ float lt_from16(uint16_t bits, int dtype) {
    return dtype == RLM_BF16 ? bf16_bits_to_float(bits) : __half2float(*reinterpret_cast<const __half*>(&bits));
}
__device__ __forceinline__ uint16_t lt_to16(float v, int dtype) {
    if (dtype == RLM_BF16) { __nv_bfloat16 h = __float2bfloat16_rn(v); return *reinterpret_cast<uint16_t*>(&h); }
    __half h = __float2half_rn(v);
    return *reinterpret_cast<uint16_t*>(&h);
}

// A stage that runs in front of the gathers, in the shared memory behind the weight slices (product
// tile, hidden tile, term and operand rows: unused until the gathers).  The standalone kernel has
// none; the whole-layer kernel runs the selector there.  A stage returns true when it has done the
// dependency wait itself (at the point its own inputs need it).
struct NoStage {
    static constexpr bool kActive = false;
    __device__ __forceinline__ bool operator()(unsigned char*, uint32_t, int, int) const { return false; }
};

// kAligned: the next LayerNorm's parameters lie on 16-byte boundaries and its rows on 8-byte ones.  Contiguous slices of
// other tensors need not; they take a build of their own, because the test in the kernel costs every launch
// instructions to fetch (a step of the 6-layer model at batch 1: 94.5 us, with the test 96.9).
template <bool kBf16, bool kAligned, typename Stage>
__device__ __forceinline__ void layer_tail_body(const CUtensorMap& map_wm, const CUtensorMap& map_w2,
                                                const LayerTailArgs& a, unsigned char* lt_smem_raw, const Stage& stage) {
    // W_m, W_2, product GEMM done, second GEMM done; partial sums, pair statistics, residual rows received
    __shared__ __align__(8) unsigned long long bars[10];         // the second GEMM has one per tile of 128 output rows
    __shared__ uint32_t tmem_base_slot;
    __shared__ int failed;
    __shared__ int pair_seq_s[kLtMaxPairs];
    __shared__ float weight_s[kLtMaxPairs];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dtype = kBf16 ? static_cast<int>(RLM_BF16) : static_cast<int>(RLM_F16);
    const uint32_t rank = lt_cluster_rank();
    const int C = a.cluster, K = a.k_out, R = a.rdim, H = a.hdim, D = a.d;
    const int s0 = blockIdx.y * a.seqs_per_cluster;
    const int nseq = min(a.n_seq - s0, a.seqs_per_cluster);
    const int pairs = nseq * K;
    const int pairs_pad = pairs <= 16 ? 16 : (pairs <= 32 ? 32 : 64);
    const int kblocks = R / kBK, chunks = R / 8, mtiles = D / kBM;
    const int h0 = static_cast<int>(rank) * kLtHC;
    const uint32_t fmt = dtype == RLM_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(pairs_pad >> 3) << 17) |
                           (static_cast<uint32_t>(kBM >> 4) << 24);

    unsigned char* base = smem_align1024(lt_smem_raw);
    const int nq_own = a.query_weight ? a.n_query / C : 0;
    const LtPlan plan = lt_plan(R, D, pairs_pad, nq_own);
    unsigned char* wm_tile = base + plan.wm;
    unsigned char* w2_tile = base + plan.w2;
    unsigned char* p_tile = base + plan.p;
    unsigned char* hid_tile = base + plan.hid;
    unsigned char* term_p = base + plan.term_p;
    unsigned char* term_a = base + plan.term_a;
    unsigned char* op_a = base + plan.op_a;
    const uint32_t p_kblock = static_cast<uint32_t>(pairs_pad) * 128u;
    // A CTA that has received all partial sums knows that every CTA is past its epilogue and its second GEMM: the
    // term rows' place receives the statistics that the CTAs push to one another, [sender][pair] of (mean, M2) over
    // the sender's 32 columns, and the hidden tile's place the residual rows [sequence][d].
    float2* stats_in = reinterpret_cast<float2*>(term_p);
    float* rows_in = reinterpret_cast<float*>(hid_tile);
    const int row_chunks = pairs_pad / 4, quads = (pairs + 3) >> 2;
    // LayerNorm parameters of this thread's owned column (column = lane), read before the dependency wait
    const int own0 = static_cast<int>(rank) * kLtOwn;
    const float pre_g = a.norm_w[own0 + lane], pre_bt = a.norm_b[own0 + lane];
    const float pre_bias = load_scalar(a.second_bias, own0 + lane, dtype);
    // warps that share a sequence at the end: warp = part x nseq + sequence
    const int my_seq = warp % nseq, part = warp / nseq, parts = (kLtThreads / 32) / nseq;
    // ... and the parameters of the next LayerNorm for the 128-column chunks part, part + parts, ... of a row
    float4 next_g[4], next_b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (part + i * parts < mtiles && part < parts) {
            next_g[i] = lt_load4<kAligned>(a.next_w + 128 * (part + i * parts) + 4 * lane);
            next_b[i] = lt_load4<kAligned>(a.next_b + 128 * (part + i * parts) + 4 * lane);
        }
    int tpo = 16;                                              // threads per projection output: 2 .. 16
    while (tpo > 2 && (nseq * nq_own * tpo > kLtThreads || (D / 8) / tpo < 2)) tpo >>= 1;
    const uint32_t wq_stride = static_cast<uint32_t>(D) * 2u + 16u * static_cast<uint32_t>(tpo);
    unsigned char* wq_tile = base + plan.wq;
    // this CTA's rows of the query-projection weight (rows padded by one 16-byte chunk per cooperating thread:
    // conflict-free reads in the projection)
    const auto request_wq = [&] {
        const int w_chunks = D / 8;
        for (int i = tid; i < nq_own * w_chunks; i += kLtThreads) {
            const int j = i / w_chunks, c = i - j * w_chunks;
            cp_async16(smem_u32(wq_tile) + j * wq_stride + 16 * c,
                       static_cast<const char*>(a.query_weight) +
                           (static_cast<size_t>(rank) * nq_own + j) * D * 2 + 16 * c);
        }
    };

    const uint32_t bar_wm = smem_u32(&bars[0]), bar_w2 = smem_u32(&bars[1]);
    const uint32_t bar_d1 = smem_u32(&bars[2]), bar_part = smem_u32(&bars[3]), bar_stat = smem_u32(&bars[4]), bar_rows = smem_u32(&bars[5]);
    const uint32_t bar_d2 = smem_u32(&bars[6]);                // + 8 per tile
    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_wm) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w2) : "memory");
        for (int i = 0; i < 10; ++i) mbar_init(smem_u32(&bars[i]), 1);
        fence_barrier_init();
        mbar_expect_tx(bar_part, static_cast<uint32_t>(C * quads) * 512u);
        mbar_expect_tx(bar_stat, static_cast<uint32_t>(C * pairs) * 8u);
        mbar_expect_tx(bar_rows, static_cast<uint32_t>(nseq * D) * 4u);
        failed = 0;
        // the weight slices do not depend on earlier kernels: requested before the dependency wait
        mbar_expect_tx(bar_wm, static_cast<uint32_t>(kblocks) * kBM * 128u);
        for (int kb = 0; kb < kblocks; ++kb)
            tma_load_2d(smem_u32(wm_tile) + kb * kBM * 128u, &map_wm, kb * kBK, h0, bar_wm);
        mbar_expect_tx(bar_w2, static_cast<uint32_t>(mtiles) * 2u * kBM * 128u);
        for (int mt = 0; mt < mtiles; ++mt)
            for (int kb = 0; kb < 2; ++kb)
                tma_load_2d(smem_u32(w2_tile) + (mt * 2 + kb) * kBM * 128u, &map_w2, h0 + kb * kBK, mt * kBM, bar_w2);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int entry = tid >> 2, quarter = tid & 3, bl = entry / K;      // bl: sequence of pair `entry`
    if (!Stage::kActive && pairs_pad == 16) request_wq();       // a parameter: before the dependency wait
    // the kernel's parameters that are first used behind the wait, into the constant cache
    asm volatile("" ::"l"(a.operand_cache), "l"(a.expanded_cache), "l"(a.anchor_index), "l"(a.partner_index), "l"(a.partner_scores),
                 "l"(a.position), "l"(a.residual), "l"(a.mix), "l"(a.normalized), "l"(a.query), "r"(a.max_t), "f"(a.eps),
                 "f"(a.next_eps));
    if (Stage::kActive) {
        // the stage's results reach the other CTAs of the cluster through global memory, ordered by
        // the cluster barrier
        if (!stage(p_tile, rank, s0, nseq)) griddep_sync();
        lt_cluster_sync();
    } else {
        griddep_sync();
    }
    if (Stage::kActive && pairs_pad == 16) request_wq();        // its place was the stage's until here
    // the residual stream was written by the previous kernel: requested now, used at the very end
    const float pre_res = a.residual[static_cast<size_t>(s0 + my_seq) * D + own0 + lane];
    const float pre_mix = *a.mix;

    // ---- gathers.  Four threads share a row to gather: they read its index themselves (one
    // broadcast load) and issue their quarter of its copies at once, so no shared-memory round
    // trip lies between the selector's indices and the first gather.  Partner operand rows go
    // straight into the swizzled product tile; copy group 0 = operand rows (needed by the
    // product GEMM), group 1 = this CTA's 128 columns of the two expanded-cache terms (needed by
    // its epilogue).  Indices and scores are all requested before the first is used, and the
    // anchors' rows are gathered by threads that a small batch's partner rows leave free.
    const size_t op_row = static_cast<size_t>(R) * 2, ex_row = static_cast<size_t>(H) * 4;
    const int a_entry = (tid - kLtThreads / 2) >> 2;          // sequence whose anchor this thread gathers
    const bool gathers_anchor = tid >= kLtThreads / 2 && a_entry < nseq;
    const int partner = entry < pairs ? a.partner_index[static_cast<size_t>(s0) * K + entry] : 0;
    const int anchor = gathers_anchor ? a.anchor_index[s0 + a_entry] : 0;
    // scores of one sequence per warp, for the softmax weights
    const int weighted = kLtThreads / 32 - 1 - warp;
    const float* score_row = a.partner_scores + static_cast<size_t>(s0 + weighted) * K;
    const float score0 = weighted < nseq && lane < K ? score_row[lane] : kNegInf;
    const float score1 = weighted < nseq && lane + 32 < K ? score_row[lane + 32] : kNegInf;
    const int t = static_cast<int>(*a.position);
    const bool bad_position = t < 0 || t >= a.max_t;          // the same in every CTA of the grid
    const int my_pair_row = min(max(partner, 0), a.max_t - 1);      // empty slots carry a sentinel that may be negative
    const int my_anchor_row = min(max(anchor, 0), a.max_t - 1);
    if (entry < pairs) {
        if (quarter == 0) pair_seq_s[entry] = bl;
        const char* src = static_cast<const char*>(a.operand_cache) +
                          (static_cast<size_t>(s0 + bl) * a.max_t + my_pair_row) * op_row;
        for (int c = quarter; c < chunks; c += 4)
            cp_async16(smem_u32(p_tile) + swizzled(entry, c, p_kblock), src + 16 * c);
    } else if (entry < pairs_pad) {
        for (int c = quarter; c < chunks; c += 4)
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};"
                         ::"r"(smem_u32(p_tile) + swizzled(entry, c, p_kblock)), "r"(0) : "memory");
    }
    if (gathers_anchor) {
        const char* src = static_cast<const char*>(a.operand_cache) +
                          (static_cast<size_t>(s0 + a_entry) * a.max_t + my_anchor_row) * op_row;
        for (int c = quarter; c < chunks; c += 4)
            cp_async16(smem_u32(op_a) + static_cast<uint32_t>(a_entry * R * 2 + 16 * c), src + 16 * c);
    }
    cp_async_commit();
    if (entry < pairs) {
        const char* src = static_cast<const char*>(a.expanded_cache) +
                          (static_cast<size_t>(s0 + bl) * a.max_t + my_pair_row) * ex_row +
                          static_cast<size_t>(H + h0) * 2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            cp_async16(smem_u32(term_p) + entry * kLtTermStride + 16 * (4 * quarter + i), src + 16 * (4 * quarter + i));
    }
    if (gathers_anchor) {
        const char* src = static_cast<const char*>(a.expanded_cache) +
                          (static_cast<size_t>(s0 + a_entry) * a.max_t + my_anchor_row) * ex_row +
                          static_cast<size_t>(h0) * 2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            cp_async16(smem_u32(term_a) + a_entry * kLtTermStride + 16 * (4 * quarter + i), src + 16 * (4 * quarter + i));
    }
    cp_async_commit();
    cp_async_wait_group1();                                    // the operand rows have arrived
    __syncthreads();
    // products o[a] * o[p], in fp32, rounded to the operand dtype, in place
    for (int i = tid; i < pairs * chunks; i += kLtThreads) {
        const int j = i / chunks, c = i - j * chunks;
        unsigned char* at = p_tile + swizzled(j, c, p_kblock);
        float pv[8], av[8];
        unpack8(*reinterpret_cast<const uint4*>(at), dtype, pv);
        unpack8(*reinterpret_cast<const uint4*>(op_a + pair_seq_s[j] * R * 2 + 16 * c), dtype, av);
        uint4 out;
        out.x = pack2(pv[0] * av[0], pv[1] * av[1], dtype);
        out.y = pack2(pv[2] * av[2], pv[3] * av[3], dtype);
        out.z = pack2(pv[4] * av[4], pv[5] * av[5], dtype);
        out.w = pack2(pv[6] * av[6], pv[7] * av[7], dtype);
        *reinterpret_cast<uint4*>(at) = out;
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot;
    const uint32_t tmem_d2 = tmem_base + 64u;                 // second GEMM: mtiles x pairs_pad columns from column 64

    // ---- product GEMM: D1[hidden column, pair] = W_m slice x products^T
    if (warp == 0) {
        const bool ok = mbar_wait(bar_wm, 0), issue = elect_lane();
        if (!ok) failed = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < kblocks; ++kb) {
            const uint64_t dw = smem_desc_sw128(smem_u32(wm_tile) + kb * kBM * 128u);
            const uint64_t dp = smem_desc_sw128(smem_u32(p_tile) + kb * p_kblock);
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                umma_f16_if(tmem_base, dw + 2 * kk, dp + 2 * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u, issue && ok);
        }
        umma_commit_if(bar_d1, issue);
    }
    __syncwarp();
    if (!mbar_wait(bar_d1, 0)) failed = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (pairs_pad == 16) { __syncwarp(); lt_cluster_arrive(); }      // the W_m slice is consumed: its place may receive
    cp_async_wait_all();                                       // the expanded-cache terms have arrived
    __syncthreads();

    // ---- epilogue of the product GEMM: + expanded-cache terms, GELU, hidden slice as the K-major
    // B tile of the second GEMM (row = pair, K = this CTA's hidden columns).  Warps 0-3 and 4-7 take
    // every other four pair columns; the columns of pairs that do not exist stay unwritten (their
    // results are never read).
    {
        const int hc = 32 * (warp & 3) + lane;                // hidden column == TMEM lane
        const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
        const unsigned char* ta = term_a + hc * 2;
        const unsigned char* tp = term_p + hc * 2;
        unsigned char* hrow = hid_tile + static_cast<uint32_t>(hc >> 6) * p_kblock + (hc & 7) * 2;
        const int hchunk = (hc >> 3) & 7;
        for (int c = 4 * (warp >> 2); c < pairs; c += 8) {
            uint32_t v[4];
            lt_tmem_ld4(tmem_base + lane_base + c, v);
            float term[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int pr = min(c + j, pairs - 1);
                term[j] = lt_from16(*reinterpret_cast<const uint16_t*>(ta + pair_seq_s[pr] * kLtTermStride), dtype) +
                          lt_from16(*reinterpret_cast<const uint16_t*>(tp + pr * kLtTermStride), dtype);
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int pr = c + j;
                *reinterpret_cast<uint16_t*>(hrow + (pr >> 3) * 1024 + (pr & 7) * 128 + ((hchunk ^ (pr & 7)) << 4)) =
                    lt_to16(gelu_tc(__uint_as_float(v[j]) + term[j]), dtype);
            }
        }
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // ---- second GEMM, split over the cluster along the hidden width:
    // D2[output row, pair] (partial) = W_2[:, this CTA's hidden columns] x hidden slice^T
    if (warp == 0) {
        const bool ok = mbar_wait(bar_w2, 0), issue = elect_lane();
        if (!ok) failed = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int mt = 0; mt < mtiles; ++mt) {
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
                const uint64_t dw = smem_desc_sw128(smem_u32(w2_tile) + (mt * 2 + kb) * kBM * 128u);
                const uint64_t dh = smem_desc_sw128(smem_u32(hid_tile) + kb * p_kblock);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk)
                    umma_f16_if(tmem_d2 + static_cast<uint32_t>(mt * pairs_pad), dw + 2 * kk, dh + 2 * kk, idesc,
                            (kb > 0 || kk > 0) ? 1u : 0u, issue && ok);
            }
            umma_commit_if(bar_d2 + 8u * mt, issue);                // each tile's partial sums leave while the next is computed
        }
    }
    __syncwarp();
    if (pairs_pad > 16) request_wq();                          // in the consumed W_m slice's place, while the GEMM runs
    cp_async_commit();
    // meanwhile the softmax weights over the active partner slots of every sequence (the last warps first: warp 0 issues)
    if (weighted < nseq) {
        int k_limit = 32 - __clz(max(t, 0) + 1);               // ceil(log2(t + 2))
        k_limit = min(max(k_limit, 1), K);
        const bool live0 = lane < k_limit && score0 > -1.0e30f, live1 = lane + 32 < k_limit && score1 > -1.0e30f;
        float mx = fmaxf(live0 ? score0 : -1.0e4f, live1 ? score1 : -1.0e4f);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float e0 = live0 ? expf(score0 - mx) : 0.0f, e1 = live1 ? expf(score1 - mx) : 0.0f;
        const float scale = 1.0f / fmaxf(warp_sum(e0 + e1), 1.0e-9f);
        if (lane < K) weight_s[weighted * K + lane] = e0 * scale;
        if (lane + 32 < K) weight_s[weighted * K + lane + 32] = e1 * scale;
    }
    if (pairs_pad > 16) {
        for (int mt = 0; mt < mtiles; ++mt)
            if (!mbar_wait(bar_d2 + 8u * mt, 0)) failed = 1;
        __syncwarp();
        lt_cluster_arrive();                                   // the W_2 slice is consumed: its place may receive
    }
    lt_cluster_wait();                                         // every CTA's receiving place is free

    // ---- reduce-scatter: the 32 output rows that a warp reads from the tensor memory belong to one CTA, which
    // receives them from every CTA of the cluster as [sender][four pairs][column][pair]: 512 contiguous bytes a store
    // of the warp, and the receiver's barrier counts them in
    unsigned char* recv = pairs_pad == 16 ? wm_tile : w2_tile;
    {
        const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
        // few pairs: by the last four warps alone, a tile behind the GEMM that warp 0 is still issuing
        const int first = pairs_pad > 16 ? warp >> 2 : warp >= 4 ? 0 : mtiles, step = pairs_pad > 16 ? 2 : 1;
        for (int mt = first; mt < mtiles; mt += step) {
            if (!mbar_wait(bar_d2 + 8u * mt, 0)) failed = 1;
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t owner = static_cast<uint32_t>(4 * mt + (warp & 3));
            const uint32_t bar = lt_peer(bar_part, owner);
            const uint32_t dst = lt_peer(smem_u32(recv), owner) + (rank * row_chunks * 32u + lane) * 16u;
            for (int c = 0; c < pairs; c += 16) {              // the accumulator has 16, 32 or 64 columns
                uint32_t v[8], w[8];
                tmem_ld8(tmem_d2 + lane_base + static_cast<uint32_t>(mt * pairs_pad + c), v);
                tmem_ld8(tmem_d2 + lane_base + static_cast<uint32_t>(mt * pairs_pad + c + 8), w);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const uint32_t at = dst + static_cast<uint32_t>(c >> 2) * 512u;
                lt_push16(at, bar, v[0], v[1], v[2], v[3]);
                if (c + 4 < pairs) lt_push16(at + 512u, bar, v[4], v[5], v[6], v[7]);
                if (c + 8 < pairs) lt_push16(at + 1024u, bar, w[0], w[1], w[2], w[3]);
                if (c + 12 < pairs) lt_push16(at + 1536u, bar, w[4], w[5], w[6], w[7]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");

    // ---- a warp owns four pairs (32 columns, a lane each): partial sums in a fixed order, so that the result does
    // not depend on timing, and (mean, M2) of the 32 columns, pushed to every CTA
    if (!mbar_wait(bar_part, 0)) failed = 1;
    float x[2][4];
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const int q = warp + 8 * it;
        if (q >= quads) break;
        const unsigned char* src = recv + (static_cast<uint32_t>(q) * 32u + lane) * 16u;
        float4 part_sum[4];                                    // senders of equal rank modulo four (C is 4, 8 or 16)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            part_sum[k] = *reinterpret_cast<const float4*>(src + static_cast<uint32_t>(k * row_chunks) * 512u);
#pragma unroll
        for (int s = 4; s < 16; s += 4) {
            if (s >= C) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 v = *reinterpret_cast<const float4*>(src + static_cast<uint32_t>((s + k) * row_chunks) * 512u);
                part_sum[k].x += v.x; part_sum[k].y += v.y; part_sum[k].z += v.z; part_sum[k].w += v.w;
            }
        }
        float4 acc;
        acc.x = (part_sum[0].x + part_sum[1].x) + (part_sum[2].x + part_sum[3].x);
        acc.y = (part_sum[0].y + part_sum[1].y) + (part_sum[2].y + part_sum[3].y);
        acc.z = (part_sum[0].z + part_sum[1].z) + (part_sum[2].z + part_sum[3].z);
        acc.w = (part_sum[0].w + part_sum[1].w) + (part_sum[2].w + part_sum[3].w);
        x[it][0] = acc.x + pre_bias; x[it][1] = acc.y + pre_bias; x[it][2] = acc.z + pre_bias; x[it][3] = acc.w + pre_bias;
        const float2 moments = lt_moments4(x[it]);
        const int pr = 4 * q + (lane >> 3);
        if (pr < pairs) {
            const uint32_t at = smem_u32(&stats_in[rank * pairs_pad + pr]);
            for (uint32_t to = lane & 7; to < static_cast<uint32_t>(C); to += 8) lt_push8(lt_peer(at, to), lt_peer(bar_stat, to), moments.x, moments.y);
        }
    }

    // ---- the pairs' statistics over the full width (equal counts: Chan's parallel variance), eight lanes a pair, and
    // the normalised pairs [pair][kLtOwnStride] for the sequences' weighted sums
    float* own_y = reinterpret_cast<float*>(base + plan.own_y);
    if (!mbar_wait(bar_stat, 0)) failed = 1;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const int q = warp + 8 * it;
        if (q >= quads) break;
        const int pr = min(4 * q + (lane >> 3), pairs - 1), from = lane & 7;
        // sums of the means' distances from the first one, of their squares and of the M2, in the same three exchanges
        const float pivot = stats_in[pr].x;
        float d1 = 0.0f, d2 = 0.0f, m2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (from + 8 * i < C) {
                const float2 st = stats_in[(from + 8 * i) * pairs_pad + pr];
                const float d = st.x - pivot;
                d1 += d;
                d2 = fmaf(d, d, d2);
                m2 += st.y;
            }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            d1 += __shfl_xor_sync(0xffffffffu, d1, o);
            d2 += __shfl_xor_sync(0xffffffffu, d2, o);
            m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        }
        const float per = 1.0f / static_cast<float>(C), mean = fmaf(d1, per, pivot);
        m2 = fmaf(static_cast<float>(kLtOwn), fmaxf(fmaf(-d1 * per, d1, d2), 0.0f), m2);
        const float rstd = rsqrtf(m2 / static_cast<float>(D) + a.eps);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float mj = __shfl_sync(0xffffffffu, mean, 8 * j), rj = __shfl_sync(0xffffffffu, rstd, 8 * j);
            if (4 * q + j < pairs) own_y[(4 * q + j) * kLtOwnStride + lane] = fmaf((x[it][j] - mj) * rj, pre_g, pre_bt);
        }
    }
    __syncthreads();
    // every warp has read its accumulators: the tensor memory goes back now, off the kernel's exit path
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }

    // ---- context and residual update: column = lane; the warps of a sequence share out the CTAs that its updated
    // columns are pushed to
    if (part < parts) {
        float ctx = 0.0f;
        for (int k0 = 0; k0 < K; k0 += 8) {
            float wk[8], y[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int at = my_seq * K + min(k0 + k, K - 1);
                wk[k] = k0 + k < K ? weight_s[at] : 0.0f;
                y[k] = own_y[at * kLtOwnStride + lane];
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) ctx = wk[k] == 0.0f ? ctx : fmaf(wk[k], y[k], ctx);     // inactive slots contribute nothing
        }
        const float hval = bad_position ? pre_res : fmaf(pre_mix, ctx, pre_res);
        if (part == 0 && !bad_position) a.residual[static_cast<size_t>(s0 + my_seq) * D + own0 + lane] = hval;
        const uint32_t at = smem_u32(&rows_in[my_seq * D + own0 + lane]);
        for (uint32_t to = part; to < static_cast<uint32_t>(C); to += parts) lt_push4(lt_peer(at, to), lt_peer(bar_rows, to), hval);
    }

    // ---- the next LayerNorm, of whole rows in every CTA: the warps of a sequence share its 128-column chunks
    cp_async_wait_all();                                       // this thread's pieces of the W_q slice
    if (!mbar_wait(bar_rows, 0)) failed = 1;
    __syncwarp();
    lt_cluster_arrive();                                       // nothing more is pushed to this CTA, nor by it
    unsigned char* rows16 = base + plan.rows;                  // [sequence][d] of 16 bits
    if (part < parts) {
        const float* row = rows_in + my_seq * D;
        // local moments of the lane's 4 mtiles columns, then five exchanges of (mean, M2) of equal halves
        float4 h[4];
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            h[i] = i < mtiles ? *reinterpret_cast<const float4*>(row + 128 * i + 4 * lane) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            sum += (h[i].x + h[i].y) + (h[i].z + h[i].w);
        }
        float count = 4.0f * static_cast<float>(mtiles), mean = sum * (1.0f / count), m2 = 0.0f;      // a power of two
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < mtiles) {
                const float dx = h[i].x - mean, dy = h[i].y - mean, dz = h[i].z - mean, dw = h[i].w - mean;
                m2 += fmaf(dx, dx, dy * dy) + fmaf(dz, dz, dw * dw);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float other = __shfl_xor_sync(0xffffffffu, mean, o), other2 = __shfl_xor_sync(0xffffffffu, m2, o), d = mean - other;
            m2 = fmaf(d * d, 0.5f * count, m2 + other2);
            mean = 0.5f * (mean + other);
            count += count;
        }
        const float rstd = rsqrtf(fmaf(m2, 1.0f / static_cast<float>(D), a.next_eps));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int chunk = part + i * parts;
            if (chunk >= mtiles) break;
            float4 v = h[0];
#pragma unroll
            for (int k = 1; k < 4; ++k)
                if (chunk == k) v = h[k];
            const float4 g = next_g[i], b = next_b[i];
            const uint2 out = make_uint2(
                pack2(fmaf((v.x - mean) * rstd, g.x, b.x), fmaf((v.y - mean) * rstd, g.y, b.y), dtype),
                pack2(fmaf((v.z - mean) * rstd, g.z, b.z), fmaf((v.w - mean) * rstd, g.w, b.w), dtype));
            const int at = 128 * chunk + 4 * lane;
            *reinterpret_cast<uint2*>(rows16 + (my_seq * D + at) * 2) = out;
            if (at / kLtOwn == static_cast<int>(rank) && !bad_position) {
                uint16_t* to = static_cast<uint16_t*>(a.normalized) + static_cast<size_t>(s0 + my_seq) * D + at;
                if (kAligned) {
                    *reinterpret_cast<uint2*>(to) = out;
                } else {
                    to[0] = static_cast<uint16_t>(out.x); to[1] = static_cast<uint16_t>(out.x >> 16);
                    to[2] = static_cast<uint16_t>(out.y); to[3] = static_cast<uint16_t>(out.y >> 16);
                }
            }
        }
    }
    __syncthreads();

    // ---- this CTA's share of the next query projection: outputs [rank * nq_own, + nq_own) of every
    // sequence, two threads per (sequence, output), fp32 accumulation
    if (nq_own > 0 && !bad_position) {
        const int n_out = nseq * nq_own, per_pass = kLtThreads / tpo, my_chunks = (D / 8) / tpo;
        const int part = tid & (tpo - 1);
        for (int o0 = 0; o0 < n_out; o0 += per_pass) {        // whole warps walk the loop together
            const int o = o0 + tid / tpo;
            const bool in = o < n_out;
            const int b = in ? o / nq_own : 0, j = in ? o - b * nq_own : 0;
            const unsigned char* wrow = wq_tile + j * wq_stride;
            const unsigned char* xrow = rows16 + (b * D) * 2;
            float acc0 = 0.0f, acc1 = 0.0f;
            for (int i = 0; i < my_chunks; i += 2) {
                float wf[8], xf[8], wg[8], xg[8];
                const int c = part + tpo * i, c2 = part + tpo * (i + 1);
                unpack8(*reinterpret_cast<const uint4*>(wrow + 16 * c), dtype, wf);
                unpack8(*reinterpret_cast<const uint4*>(xrow + 16 * c), dtype, xf);
                unpack8(*reinterpret_cast<const uint4*>(wrow + 16 * c2), dtype, wg);
                unpack8(*reinterpret_cast<const uint4*>(xrow + 16 * c2), dtype, xg);
#pragma unroll
                for (int e = 0; e < 8; ++e) { acc0 = fmaf(wf[e], xf[e], acc0); acc1 = fmaf(wg[e], xg[e], acc1); }
            }
            float acc = acc0 + acc1;
            for (int sh = 1; sh < tpo; sh <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
            if (in && part == 0)
                static_cast<uint16_t*>(a.query)[static_cast<size_t>(s0 + b) * a.n_query + rank * nq_own + j] = lt_to16(acc, dtype);
        }
    }
    __syncwarp();
    lt_cluster_wait();                                         // no CTA leaves while another may still push to it
    if (tid == 0 && a.status) {
        if (*reinterpret_cast<volatile int*>(&failed)) atomicOr(a.status, RLM_DEV_TIMEOUT);
        if (bad_position) atomicOr(a.status, RLM_DEV_POSITION);
    }
}

inline bool lt_aligned(const LayerTailArgs& a) {
    return aligned16(a.next_w) && aligned16(a.next_b) && (reinterpret_cast<uintptr_t>(a.normalized) & 7u) == 0;
}

int lt_validate(const LayerTailArgs& a) {
    if (a.n_seq < 1 || a.k_out < 1 || a.k_out > kLtMaxPairs || a.max_t < 1) {
        set_error("relation_layer_tail: sizes must be positive and K at most 64");
        return RLM_ERR_SHAPE;
    }
    if (a.dtype != RLM_BF16 && a.dtype != RLM_F16) {
        set_error("relation_layer_tail: caches and weights must share bfloat16 or float16");
        return RLM_ERR_UNSUPPORTED;
    }
    if (a.hdim % kLtHC != 0 || (a.hdim / kLtHC != 4 && a.hdim / kLtHC != 8 && a.hdim / kLtHC != 16) ||
        a.d % kBM != 0 || a.d > 512 || a.d / (a.hdim / kLtHC) != kLtOwn || a.rdim % kBK != 0 || a.rdim > 256) {
        set_error("relation_layer_tail: needs H = 4 d with d in {128, 256, 512} and R a multiple of 64 up to 256");
        return RLM_ERR_UNSUPPORTED;
    }
    const int cluster = a.hdim / kLtHC;
    if (a.query_weight && (a.n_query < cluster || a.n_query % (16 * cluster) != 0 || a.n_query / cluster > 64 || !a.query ||
                           static_cast<size_t>(a.n_query / cluster) * (a.d * 2 + 256) > static_cast<size_t>(a.rdim / kBK) * kBM * 128)) {
        set_error("relation_layer_tail: query projection width must be a multiple of 16 outputs per CTA (H / 128 CTAs), at most 64 each");
        return RLM_ERR_UNSUPPORTED;
    }
    if (lt_smem_bytes(a.rdim, a.d, a.query_weight ? a.n_query / cluster : 0) > static_cast<uint32_t>(kSmemDynamicLimit)) {
        set_error("relation_layer_tail: the weight slices exceed 227 KB of shared memory");
        return RLM_ERR_SMEM;
    }
    return RLM_OK;
}

int lt_prepare(const void* kernel, int cluster) {
    // clusters of more than 8 CTAs are an opt-in of every kernel, on every device
    static std::mutex guard;
    static const void* done_kernel[64 * 4] = {};
    static int done_device[64 * 4] = {};
    static int done_count = 0;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) { cudaGetLastError(); return RLM_ERR_LAUNCH; }
    int rc = allow_large_smem(kernel, kSmemPerCta);
    if (rc != RLM_OK) return rc;
    std::lock_guard<std::mutex> lock(guard);
    for (int i = 0; i < done_count; ++i)
        if (done_kernel[i] == kernel && done_device[i] == device) return RLM_OK;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        set_error("relation_layer_tail: clusters of 16 CTAs are not available on this device");
        return RLM_ERR_UNSUPPORTED;
    }
    if (done_count < 64 * 4) {
        done_kernel[done_count] = kernel;
        done_device[done_count] = device;
        ++done_count;
    }
    (void)cluster;
    return RLM_OK;
}


}  // namespace
}  // namespace rlm

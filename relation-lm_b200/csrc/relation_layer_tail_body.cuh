// Body of the relation layer tail (see relation_layer_tail.cu for the description) and its host-side
// helpers, shared by the standalone kernel and by the whole-layer kernel that runs the selector
// in front of it (relation_select.cu).
#pragma once

#include <mutex>

#include "rlm_tcgen05.cuh"

namespace rlm {
namespace {

constexpr int kLtThreads = 256;
constexpr int kLtHC = 128;            // hidden columns per CTA (192 at d = 768)
constexpr int kLtMaxPairs = 64;       // (sequence, partner) pairs per cluster
constexpr int kLtMaxSeq = 8;          // sequences per cluster
constexpr int kLtOwn = 32;            // output columns a CTA owns after the reduce-scatter (d / C; 48 at d = 768)
constexpr uint32_t kLtW2Tile = kBM * 128u;           // 128 output rows x 64 hidden columns
constexpr int kLtMaxRing = 10;        // W_2 tiles in flight where the slice is streamed

// d = 768: 16 CTAs of 192 hidden and 48 output columns, whose W_2 slice is streamed; otherwise H / 128 CTAs.
__host__ __device__ inline bool lt_wide(int d) { return d > 512; }
__host__ __device__ inline int lt_hidden(int d) { return lt_wide(d) ? 192 : kLtHC; }
__host__ __device__ inline int lt_cluster(int d) { return 4 * d / lt_hidden(d); }
__host__ __device__ inline int lt_owned(int d) { return lt_wide(d) ? 48 : kLtOwn; }

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
    uint32_t wm, w2, p, hid, term_p, term_a, stats_out, wq, total;
    uint32_t own_y, rows, rows_in;       // later uses of p, w2 and hid: see lt_plan
    int ring;                            // W_2 tiles in flight (wide: the slice has 18)
};

// Launches of more than 16 pairs a cluster.
__host__ __device__ inline bool lt_many(int seqs_per_cluster, int k_out) { return seqs_per_cluster * k_out > 16; }
// CTAs that share their hidden slices and divide the output rows (neighbours in the cluster): see relation_layer_tail.cu.
// The partial sums of few pairs are too short for that (us a step of 6 layers of d 512, batch 1 and 8: 84.0 and 94.6
// without, 84.0 and 94.5 with it; of 4 layers of d 256, batch 1: 57.5, 59.4).
__host__ __device__ inline int lt_sharing(int d, bool many) { return lt_wide(d) || (d >= 2 * kBM && many) ? 2 : 1; }

// The partial sums that a CTA receives, [sender][four pairs][owned column][pair] of 512 d pairs / 128 bytes (half of it from
// sharing CTAs) in all, take the place of a consumed weight slice: W_m's for 16 pairs, W_2's for more (the W_q slice then
// waits for W_m's).  nq_own: rows of the query-projection weight per CTA.
__host__ __device__ inline LtPlan lt_plan(int rdim, int d, bool many, int pairs_pad, int nq_own) {
    LtPlan p;
    const bool wide = lt_wide(d);
    const uint32_t hc = lt_hidden(d), own = lt_owned(d), term_stride = 2u * hc + 16u;
    uint32_t off = 0;
    const uint32_t received = 4u * static_cast<uint32_t>(d) * pairs_pad / lt_sharing(d, many);
    p.wm = off;     off += static_cast<uint32_t>(rdim / kBK) * hc * 128u;            // W_m slice
    if (pairs_pad == 16 && off < received) off = received;
    p.w2 = off;     if (!wide) off += static_cast<uint32_t>(d / kBM) * 2u * kLtW2Tile;      // W_2 slice (wide: at the end)
    // product tile; later this CTA's hidden slice, which is written when the product GEMM is done; later the normalised pairs
    const uint32_t product = static_cast<uint32_t>(rdim / kBK) * pairs_pad * 128u, slice = hc / kBK * pairs_pad * 128u;
    const uint32_t normalised = pairs_pad * (own + 1u) * 4u, rows_in = static_cast<uint32_t>(kLtMaxSeq) * d * 4u;
    p.p = off;      off += product > slice ? product : slice;
    if (off - p.p < normalised) off = p.p + normalised;
    off = (off + 1023u) & ~1023u;
    p.hid = p.rows_in = off; off += slice;                                           // the sharing CTA's slice; later the residual rows
    if (!wide && off - p.hid < rows_in) off = p.hid + rows_in;
    p.term_p = off; off += pairs_pad * term_stride;
    p.term_a = off; off += kLtMaxSeq * term_stride;
    p.stats_out = off; off += kLtMaxPairs * 8u;
    p.wq = p.wm;
    // The last LayerNorm's rows take W_2's place, not the normalised pairs': a warp may write its rows while another
    // of its CTA still sums its pairs (the barrier between them counts what this CTA is sent, and only one warp a
    // sequence sends to it).  W_2's place is free in every warp by then: the statistics that a CTA waits for include
    // its own, and those follow its second GEMM and its reads of the partial sums.
    p.own_y = p.p;
    p.ring = 0;
    if (wide) {
        // the ring takes what is left; in its place, later: the residual rows that come in, the last LayerNorm's rows and,
        // where W_m's place receives the partial sums, the W_q slice
        p.w2 = (off + 1023u) & ~1023u;
        const int left = kSmemDynamicLimit - 1024 - static_cast<int>(p.w2);
        p.ring = left < 0 ? 0 : left / static_cast<int>(kLtW2Tile);
        if (p.ring > kLtMaxRing) p.ring = kLtMaxRing;
        off = p.w2 + p.ring * kLtW2Tile;
        p.rows_in = p.w2;
        p.rows = p.w2 + rows_in;
        if (pairs_pad == 16) p.wq = p.rows + rows_in / 2;
    } else {
        if (pairs_pad == 16) { p.wq = off; off += static_cast<uint32_t>(nq_own) * (2u * d + 256u); }
        p.rows = p.w2;
    }
    p.total = off;
    return p;
}

// Dynamic shared memory of a launch, whatever its pairs per cluster.
inline uint32_t lt_smem_bytes(int rdim, int d, int nq_own) {
    uint32_t most = 0;
    for (int pairs = 16; pairs <= kLtMaxPairs; pairs *= 2)
        for (int many = pairs > 16; many < 2; ++many) {
            const uint32_t total = lt_plan(rdim, d, many, pairs, nq_own).total;
            if (total > most) most = total;
        }
    return most + 1024;
}

// Dynamic shared memory of a whole-layer launch, whose stage needs `stage` bytes behind the weight slices.
inline uint32_t lt_smem_bytes_with_stage(int rdim, int d, int nq_own, int stage) {
    uint32_t most = lt_smem_bytes(rdim, d, nq_own);
    for (int pairs = 16; pairs <= kLtMaxPairs; pairs *= 2) {
        const uint32_t total = lt_plan(rdim, d, pairs > 16, pairs, nq_own).p + static_cast<uint32_t>(stage) + 1024u;
        if (total > most) most = total;
    }
    return most;
}

// Bytes that a stage in front of the gathers may take: 64 pairs' product tile, the residual rows or hidden slice, the terms and
// eight sequences' operand rows (which once stood there; what fitted then fits: a launch's shared memory counts the stage).
inline int lt_stage_room(int rdim, int d) {
    const int product = rdim / kBK * kLtMaxPairs * 128, normalised = kLtMaxPairs * (kLtOwn + 1) * 4;
    const int slice = 2 * kLtMaxPairs * 128, rows_in = kLtMaxSeq * d * 4;
    return (((product > normalised ? product : normalised) + 1023) & ~1023) + (slice > rows_in ? slice : rows_in) +
           (kLtMaxPairs + kLtMaxSeq) * (2 * kLtHC + 16) + kLtMaxSeq * rdim * 2;
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
__device__ __forceinline__ void lt_copy_cluster(uint32_t remote_dst, uint32_t src, uint32_t bytes, uint32_t remote_bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(remote_dst), "r"(src), "r"(bytes), "r"(remote_bar) : "memory");
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

// The same over a half-warp's 16 lanes of three columns each, x[column][j], for j = (lane % 16) / 4.
__device__ __forceinline__ float2 lt_moments4(const float (&x)[3][4]) {
    const bool hi = threadIdx.x & 8, mid = threadIdx.x & 4;
    float m4[4], v4[4], m[2], v[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        m4[j] = (x[0][j] + x[1][j] + x[2][j]) * (1.0f / 3.0f);
        const float d0 = x[0][j] - m4[j], d1 = x[1][j] - m4[j], d2 = x[2][j] - m4[j];
        v4[j] = fmaf(d0, d0, fmaf(d1, d1, d2 * d2));
    }
    float count = 3.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, hi ? m4[j] : m4[2 + j], 8), other2 = __shfl_xor_sync(0xffffffffu, hi ? v4[j] : v4[2 + j], 8);
        const float mine = hi ? m4[2 + j] : m4[j], d = mine - other;
        m[j] = 0.5f * (mine + other);
        v[j] = fmaf(d * d, 0.5f * count, (hi ? v4[2 + j] : v4[j]) + other2);
    }
    count += count;
    float mean = mid ? m[1] : m[0], m2 = mid ? v[1] : v[0];
    float give_mean = mid ? m[0] : m[1], give_m2 = mid ? v[0] : v[1];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
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
template <bool kBf16, bool kAligned, bool kWide, bool kMany, typename Stage>
__device__ __forceinline__ void layer_tail_body(const CUtensorMap& map_wm, const CUtensorMap& map_w2,
                                                const LayerTailArgs& a, unsigned char* lt_smem_raw, const Stage& stage) {
    // W_m, W_2 (own columns), product GEMM done; partial sums, pair statistics, residual rows, shared slice received; W_2 (the
    // sharing CTA's columns)
    __shared__ __align__(8) unsigned long long bars[12 + (kWide ? 2 * kLtMaxRing : 0)];      // behind them one per tile of 128 output rows: second GEMM done
    constexpr int kHC = kWide ? 192 : kLtHC, kOwn = kWide ? 48 : kLtOwn, kOwnStride = kOwn + 1, kSlices = kHC / kBK;
    constexpr uint32_t kTermStride = 2 * kHC + 16;               // padded row of the staged expanded-cache terms
    constexpr int kChunks128 = kWide ? 6 : 4;                    // most 128-column chunks of a row
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
    const int pairs_pad = !kMany || pairs <= 16 ? 16 : (pairs <= 32 ? 32 : 64);
    const int kblocks = R / kBK, chunks = R / 8, mtiles = (D / (kWide || kMany ? lt_sharing(D, kMany) : 1)) / kBM, row_tiles = D / kBM;
    const int h0 = static_cast<int>(rank) * kHC;
    // this CTA's half of the output rows (g), its place among the CTAs of that half, the CTA that it shares with
    const int share = kWide ? 2 : kMany ? lt_sharing(D, true) : 1, gs = share - 1, g = static_cast<int>(rank) & gs, place = static_cast<int>(rank) >> gs;
    const int d_rows = D >> gs, senders = C >> gs;
    const uint32_t sharer = rank ^ static_cast<uint32_t>(gs);
    const uint32_t fmt = dtype == RLM_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(pairs_pad >> 3) << 17) |
                           (static_cast<uint32_t>(kBM >> 4) << 24);

    unsigned char* base = smem_align1024(lt_smem_raw);
    const int nq_own = a.query_weight ? a.n_query / C : 0;
    const LtPlan plan = lt_plan(R, D, kMany, pairs_pad, nq_own);
    unsigned char* wm_tile = base + plan.wm;
    unsigned char* w2_tile = base + plan.w2;
    unsigned char* p_tile = base + plan.p;
    unsigned char* hid_tile = base + plan.hid;
    unsigned char* term_p = base + plan.term_p;
    unsigned char* term_a = base + plan.term_a;
    float2* stats_out = reinterpret_cast<float2*>(base + plan.stats_out);      // this CTA's [pair] (mean, M2)
    const uint32_t p_kblock = static_cast<uint32_t>(pairs_pad) * 128u;
    // A CTA that has received all partial sums knows that every CTA is past its epilogue and its second GEMM: the
    // term rows' place receives the statistics that the CTAs push to one another, [sender][pair] of (mean, M2) over
    // the sender's columns, and the shared slice's place (or W_2's) the residual rows [sequence][d].
    float2* stats_in = reinterpret_cast<float2*>(term_p);
    float* rows_in = reinterpret_cast<float*>(base + plan.rows_in);
    const int row_chunks = pairs_pad / 4, quads = (pairs + 3) >> 2;
    // LayerNorm parameters of this thread's owned columns, read before the dependency wait
    const int own0 = g * d_rows + place * kOwn;
    // (wide: a half-warp has the owned columns, three to a lane)
    const int column = kWide ? lane & 15 : lane;
    constexpr int kOwnPer = kWide ? 3 : 1;
    float pre_g[kOwnPer], pre_bt[kOwnPer], pre_bias[kOwnPer];
#pragma unroll
    for (int i = 0; i < kOwnPer; ++i) {
        pre_g[i] = a.norm_w[own0 + column + 16 * i];
        pre_bt[i] = a.norm_b[own0 + column + 16 * i];
        pre_bias[i] = load_scalar(a.second_bias, own0 + column + 16 * i, dtype);
    }
    // warps that share a sequence at the end: warp = part x nseq + sequence
    const int my_seq = warp % nseq, part = warp / nseq, parts = (kLtThreads / 32) / nseq;
    // ... and the parameters of the next LayerNorm for the 128-column chunks part, part + parts, ... of a row
    float4 next_g[kChunks128], next_b[kChunks128];
#pragma unroll
    for (int i = 0; i < kChunks128; ++i)
        if (part + i * parts < row_tiles && part < parts) {
            next_g[i] = lt_load4<kAligned>(a.next_w + 128 * (part + i * parts) + 4 * lane);
            next_b[i] = lt_load4<kAligned>(a.next_b + 128 * (part + i * parts) + 4 * lane);
        }
    const float per = 1.0f / static_cast<float>(C), inv_d = 1.0f / static_cast<float>(D);
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
    const uint32_t bar_hid = smem_u32(&bars[6]), bar_w2b = smem_u32(&bars[7]);
    const uint32_t bar_d2 = smem_u32(&bars[8]);                // + 8 per tile
    // wide: W_2's tiles n = ([this CTA's, the sharing CTA's][K-block][tile_at(i)]) go through a ring
    const int ring = plan.ring;
    const auto bar_full = [&](int slot) { return smem_u32(&bars[12 + (kWide ? slot : 0)]); };
    const auto bar_empty = [&](int slot) { return smem_u32(&bars[12 + (kWide ? kLtMaxRing + slot : 0)]); };
    // The CTAs take the tiles of output rows in different orders, so that their partial sums go to all CTAs at any
    // time: in one order, four of sixteen received and the last ones' sums came late.
    const auto tile_at = [&](int i) { return kWide ? (i + place) % 3 : (i + place) & (mtiles - 1); };
    const auto request_w2 = [&](int n) {
        const int other = n / 9, kb = n / 3 - 3 * other, mt = tile_at(n % 3), slot = n % ring;
        mbar_expect_tx(bar_full(slot), kLtW2Tile);
        tma_load_2d(smem_u32(w2_tile) + slot * kLtW2Tile, &map_w2, (other ? static_cast<int>(sharer) : static_cast<int>(rank)) * kHC + kb * kBK,
                    g * d_rows + mt * kBM, bar_full(slot));
    };
    const uint32_t slice_rows = static_cast<uint32_t>((pairs + 7) & ~7) * 128u;          // bytes of a K-block that hold pairs
    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_wm) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w2) : "memory");
        for (int i = 0; i < 12 + (kWide ? 2 * kLtMaxRing : 0); ++i) mbar_init(smem_u32(&bars[i]), kWide && i == 2 ? 2 : 1);
        fence_barrier_init();
        mbar_expect_tx(bar_part, static_cast<uint32_t>(senders * quads) * (kOwn * 16u));
        mbar_expect_tx(bar_stat, static_cast<uint32_t>(C * ((pairs + 1) & ~1)) * 8u);
        mbar_expect_tx(bar_rows, static_cast<uint32_t>(nseq * D) * 4u);
        failed = 0;
        // the weight slices do not depend on earlier kernels: requested before the dependency wait
        mbar_expect_tx(bar_wm, static_cast<uint32_t>(kblocks) * kHC * 128u);
        for (int kb = 0; kb < kblocks; ++kb)
            tma_load_2d(smem_u32(wm_tile) + kb * kHC * 128u, &map_wm, kb * kBK, h0, bar_wm);
        // W_2: this half's output rows, by K-block of hidden columns: this CTA's two, then the sharing CTA's
        if (kWide)
            for (int n = 0; n < ring - 1; ++n) request_w2(n);   // (the last place holds the products' low parts first)
        for (int other = 0; !kWide && other < share; ++other) {
            const uint32_t bar = other ? bar_w2b : bar_w2;
            const int from = (other ? static_cast<int>(sharer) : static_cast<int>(rank)) * kLtHC;
            mbar_expect_tx(bar, static_cast<uint32_t>(mtiles) * 2u * kBM * 128u);
            for (int kb = 0; kb < 2; ++kb)
                for (int mt = 0; mt < mtiles; ++mt)
                    tma_load_2d(smem_u32(w2_tile) + ((2 * other + kb) * mtiles + mt) * kBM * 128u, &map_w2, from + kb * kBK,
                                g * d_rows + mt * kBM, bar);
        }
        if (share > 1) mbar_expect_tx(bar_hid, kSlices * slice_rows);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (kWide || kMany) {                                      // every CTA's barriers are initialised (few: see the next barrier)
        __syncwarp();
        lt_cluster_sync();
    }
    // the threads of a pair (16, 8 or 4), this thread's place among them, the pair's sequence
    const int tpp_shift = pairs_pad == 16 ? 4 : pairs_pad == 32 ? 3 : 2, tpp = 1 << tpp_shift;
    const int entry = tid >> tpp_shift, sub = tid & (tpp - 1), bl = entry / K, quarter = tid & 3;
    if (!kWide && !Stage::kActive && pairs_pad == 16) request_wq();       // a parameter: before the dependency wait
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
    constexpr int kResPer = kWide ? 2 : 1;
    float pre_res[kResPer];
#pragma unroll
    for (int i = 0; i < kResPer; ++i) pre_res[i] = a.residual[static_cast<size_t>(s0 + my_seq) * D + own0 + min(lane + 32 * i, kOwn - 1)];
    const float pre_mix = *a.mix;

    // ---- gathers.  Some threads share a pair: they read its two indices themselves (broadcast loads) and request their
    // parts of its operand rows into registers at once, so that neither a shared-memory round trip nor a barrier lies
    // between the selector's indices and the products, which go straight into the swizzled tile.  Behind them, by
    // cp.async, this CTA's columns of the two expanded-cache terms, needed by the epilogue.  (Operand rows by cp.async,
    // multiplied in place behind a barrier: 2 850 cycles from the wait to the products at batch 1, now 1 550.)  The scores are
    // requested with the indices; the anchors' terms are gathered by threads that a small batch's pairs leave free.
    const size_t op_row = static_cast<size_t>(R) * 2, ex_row = static_cast<size_t>(H) * 4;
    const int a_entry = (tid - kLtThreads / 2) >> 2;          // sequence whose anchor's terms this thread gathers
    const bool gathers_anchor = tid >= kLtThreads / 2 && a_entry < nseq;
    const int partner = entry < pairs ? a.partner_index[static_cast<size_t>(s0) * K + entry] : 0;
    const int pair_anchor = entry < pairs ? a.anchor_index[s0 + bl] : 0;
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
    const size_t seq_row = static_cast<size_t>(s0 + bl) * a.max_t;
    const uint4* partner_op = reinterpret_cast<const uint4*>(static_cast<const char*>(a.operand_cache) + (seq_row + my_pair_row) * op_row) + sub;
    const uint4* anchor_op = reinterpret_cast<const uint4*>(static_cast<const char*>(a.operand_cache) + (seq_row + min(max(pair_anchor, 0), a.max_t - 1)) * op_row) + sub;
    uint4 pv[4], av[4];                                        // four chunks of a row at a time
    const auto request = [&](int c0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool in = entry < pairs && c0 + tpp * i + sub < chunks;
            pv[i] = in ? partner_op[c0 + tpp * i] : make_uint4(0, 0, 0, 0);
            av[i] = in ? anchor_op[c0 + tpp * i] : make_uint4(0, 0, 0, 0);
        }
    };
    request(0);
    if (entry < pairs) {
        if (sub == 0) pair_seq_s[entry] = bl;
        const char* src = static_cast<const char*>(a.expanded_cache) + (seq_row + my_pair_row) * ex_row + static_cast<size_t>(H + h0) * 2;
#pragma unroll
        for (int i = 0; i < kHC / 32; ++i)
            if (sub + tpp * i < kHC / 8) cp_async16(smem_u32(term_p) + entry * kTermStride + 16 * (sub + tpp * i), src + 16 * (sub + tpp * i));
    }
    if (gathers_anchor) {
        const char* src = static_cast<const char*>(a.expanded_cache) +
                          (static_cast<size_t>(s0 + a_entry) * a.max_t + my_anchor_row) * ex_row +
                          static_cast<size_t>(h0) * 2;
#pragma unroll
        for (int i = 0; i < kHC / 32; ++i)
            cp_async16(smem_u32(term_a) + a_entry * kTermStride + 16 * (kHC / 32 * quarter + i), src + 16 * (kHC / 32 * quarter + i));
    }
    cp_async_commit();
    // products o[a] * o[p], in fp32, rounded to the operand dtype; zeros in the rows of pairs that do not exist.  Wide: the
    // difference to the rounded product in a tile of its own, with which the product GEMM has all bits of the product
    // (16 of two bfloat16 factors, 22 of two halves), as the separate kernels below 256 pairs have it.
    const uint32_t low_tile = smem_u32(w2_tile) + static_cast<uint32_t>(kWide ? ring - 1 : 0) * kLtW2Tile;
    for (int c0 = 0;;) {
        if (entry < pairs_pad)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (c0 + tpp * i + sub >= chunks) break;
                float fp[8], fa[8];
                unpack8(pv[i], dtype, fp);
                unpack8(av[i], dtype, fa);
                const uint32_t at = swizzled(entry, c0 + tpp * i + sub, p_kblock);
                uint32_t high[4], low[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float x = fp[2 * e] * fa[2 * e], y = fp[2 * e + 1] * fa[2 * e + 1];
                    high[e] = pack2(x, y, dtype);
                    if (kWide) {
                        const float hx = lt_from16(static_cast<uint16_t>(high[e]), dtype), hy = lt_from16(static_cast<uint16_t>(high[e] >> 16), dtype);
                        low[e] = pack2(isfinite(hx) ? x - hx : 0.0f, isfinite(hy) ? y - hy : 0.0f, dtype);
                    }
                }
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                             ::"r"(smem_u32(p_tile) + at), "r"(high[0]), "r"(high[1]), "r"(high[2]), "r"(high[3]) : "memory");
                if (kWide)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                 ::"r"(low_tile + at), "r"(low[0]), "r"(low[1]), "r"(low[2]), "r"(low[3]) : "memory");
            }
        c0 += 4 * tpp;
        if (c0 >= chunks) break;
        request(c0);
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot;
    const uint32_t tmem_d2 = tmem_base + (kWide ? 128u : 64u);      // second GEMM: mtiles x pairs_pad columns

    // ---- product GEMM: D1[hidden column, pair] = W_m slice x products^T
    // (wide: 192 hidden columns as two overlapping tiles of 128, rows 0 .. 127 and rows 64 .. 191, a warp each)
    if (warp < (kWide ? 2 : 1)) {
        const bool ok = mbar_wait(bar_wm, 0), issue = elect_lane();
        if (!ok) failed = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tile = kWide ? static_cast<uint32_t>(warp) : 0u;
        for (int kb = 0; kb < kblocks; ++kb) {
            const uint64_t dw = smem_desc_sw128(smem_u32(wm_tile) + kb * kHC * 128u) + tile * (64 * 128 >> 4);
#pragma unroll
            for (int part = 0; part < (kWide ? 2 : 1); ++part) {
                const uint64_t dp = smem_desc_sw128((part ? low_tile : smem_u32(p_tile)) + kb * p_kblock);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk)
                    umma_f16_if(tmem_base + 64u * tile, dw + 2 * kk, dp + 2 * kk, idesc, (kb > 0 || part > 0 || kk > 0) ? 1u : 0u, issue && ok);
            }
        }
        umma_commit_if(bar_d1, issue);
    }
    __syncwarp();
    cp_async_wait_all();                                       // the expanded-cache terms have arrived
    __syncthreads();

    // ---- epilogue of the product GEMM: + expanded-cache terms, GELU, hidden slice as the K-major
    // B tile of the second GEMM (row = pair, K = this CTA's hidden columns).  Warps 0-3 and 4-7 take
    // every other four pair columns; the columns of pairs that do not exist stay unwritten (their
    // results are never read).  The terms of the first eight pairs are added up while the GEMM runs.
    {
        const int quadrant = warp & 3;
        const uint32_t lane_base = static_cast<uint32_t>(32 * quadrant) << 16;
        float term[8];
        uint32_t ta, tp;
        unsigned char* hrow;
        int hchunk;
        const auto at_column = [&](int hc) {                  // this thread's hidden column
            ta = smem_u32(term_a) + hc * 2;
            tp = smem_u32(term_p) + hc * 2;
            hrow = p_tile + static_cast<uint32_t>(hc >> 6) * p_kblock + (hc & 7) * 2;
            hchunk = (hc >> 3) & 7;
        };
        const auto terms = [&](int c, int step) {             // of pairs c .. c + 3 and c + step .. c + step + 3
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int pr = min(c + (j & 3) + (j & 4 ? step : 0), pairs - 1);
                uint16_t from_a, from_p;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(from_a) : "r"(ta + pair_seq_s[pr] * kTermStride));
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(from_p) : "r"(tp + pr * kTermStride));
                term[j] = lt_from16(from_a, dtype) + lt_from16(from_p, dtype);
            }
        };
        const auto finish = [&](uint32_t from, int c, int step) {      // fours of pairs c, c + step, .. of the accumulator at `from`
            for (; c < pairs; c += 2 * step) {
                uint32_t v[8];
                lt_tmem_ld4(from + lane_base + c, *reinterpret_cast<uint32_t(*)[4]>(&v[0]));
                if (c + step < pairs) lt_tmem_ld4(from + lane_base + c + step, *reinterpret_cast<uint32_t(*)[4]>(&v[4]));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const auto store = [&](int pr, float h) {
                    *reinterpret_cast<uint16_t*>(hrow + (pr >> 3) * 1024 + (pr & 7) * 128 + ((hchunk ^ (pr & 7)) << 4)) = lt_to16(h, dtype);
                };
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    if (j >= 4 && c + step >= pairs) break;
                    const int pr = c + (j & 3) + (j & 4 ? step : 0);
                    // (the two are different pairs, perhaps of different sequences: a reciprocal each)
                    const float2 h = gelu_tc2(make_float2(__uint_as_float(v[j]) + term[j], __uint_as_float(v[j + 1]) + term[j + 1]));
                    store(pr, h.x);
                    store(pr + 1, h.y);
                }
                if (c + 2 * step < pairs) terms(c + 2 * step, step);
            }
        };
        // Wide: quadrants 0, 1 have columns 0 .. 63 in the first tile, quadrants 2, 3 columns 128 .. 191 in the second; of
        // columns 64 .. 127, which both tiles hold, every quadrant of the four takes every fourth four of pairs.
        const bool upper = kWide && quadrant >= 2;
        at_column(32 * quadrant + lane + (upper ? 64 : 0));
        terms(4 * (warp >> 2), 8);
        if (!mbar_wait(bar_d1, 0)) failed = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (pairs_pad == 16) { __syncwarp(); lt_cluster_arrive(); }      // the W_m slice is consumed: its place may receive
        finish(tmem_base + (upper ? 64u : 0u), 4 * (warp >> 2), 8);
        if (kWide) {
            const int first = 4 * ((warp >> 2) + (upper ? 2 : 0));
            at_column(64 + 32 * (quadrant & 1) + lane);
            if (first < pairs) terms(first, 16);
            finish(tmem_base + (upper ? 0u : 64u), first, 16);
        }
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // ---- second GEMM, split over the cluster along the hidden width:
    // D2[output row, pair] (partial) = W_2[:, this CTA's hidden columns] x hidden slice^T
    // (by two warps: one issues an instruction every 50 cycles, a narrow one takes 32)
    // The sharing CTA's slice is on its way while this CTA's own is multiplied.
    if (share > 1 && tid == 32 * 2)
        for (int kb = 0; kb < kSlices; ++kb)
            lt_copy_cluster(lt_peer(smem_u32(hid_tile) + kb * p_kblock, sharer), smem_u32(p_tile) + kb * p_kblock, slice_rows, lt_peer(bar_hid, sharer));
    if (kWide) {
        if (warp == 0 || warp == 1 || warp == 3) {             // a tile of output rows each
            const int i = warp == 3 ? 2 : warp, mt = tile_at(i);
            const bool issue = elect_lane();
            bool ok = true;
            for (int n = i; n < 18; n += 3) {
                const int other = n / 9, kb = n / 3 - 3 * other, slot = n % ring;
                if (n == 9 + i) ok = mbar_wait(bar_hid, 0) && ok;
                ok = mbar_wait(bar_full(slot), (n / ring) & 1) && ok;
                if (!ok) failed = 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t dw = smem_desc_sw128(smem_u32(w2_tile) + slot * kLtW2Tile);
                const uint64_t dh = smem_desc_sw128(smem_u32(other ? hid_tile : p_tile) + kb * p_kblock);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk)
                    umma_f16_if(tmem_d2 + static_cast<uint32_t>(mt * pairs_pad), dw + 2 * kk, dh + 2 * kk, idesc, (n > i || kk > 0) ? 1u : 0u, issue && ok);
                umma_commit_if(bar_empty(slot), issue);
            }
            umma_commit_if(bar_d2 + 8u * mt, issue);
        } else if (warp == 2 && lane == 0) {
            request_w2(ring - 1);                              // the low parts are consumed
            for (int n = ring; n < 18; ++n) {
                if (!mbar_wait(bar_empty(n % ring), (n / ring - 1) & 1)) { failed = 1; break; }
                request_w2(n);
            }
        }
    } else if (warp < 2) {
        const bool issue = elect_lane();
        bool ok = true;
        for (int other = 0; other < share; ++other) {
            ok = mbar_wait(other ? bar_w2b : bar_w2, 0) && (!other || mbar_wait(bar_hid, 0)) && ok;
            if (!ok) failed = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t slice = smem_u32(other ? hid_tile : p_tile);
            for (int i = warp; i < mtiles; i += 2) {
                const int mt = tile_at(i);
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    const uint64_t dw = smem_desc_sw128(smem_u32(w2_tile) + ((2 * other + kb) * mtiles + mt) * kBM * 128u);
                    const uint64_t dh = smem_desc_sw128(slice + kb * p_kblock);
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)
                        umma_f16_if(tmem_d2 + static_cast<uint32_t>(mt * pairs_pad), dw + 2 * kk, dh + 2 * kk, idesc,
                                (other > 0 || kb > 0 || kk > 0) ? 1u : 0u, issue && ok);
                }
                if (other + 1 == share) umma_commit_if(bar_d2 + 8u * mt, issue);      // each tile's partial sums leave while the next is computed
            }
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
        // few pairs in four tiles: by the last four warps alone, a tile behind the GEMM that the first two are still issuing
        const bool behind = share == 1 && pairs_pad == 16;
        for (int i = behind ? (warp >= 4 ? 0 : mtiles) : warp >> 2; i < mtiles; i += behind ? 1 : 2) {
            const int mt = tile_at(i);
            if (!mbar_wait(bar_d2 + 8u * mt, 0)) failed = 1;
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = mt * kBM + 32 * (warp & 3) + lane, owner_place = row / kOwn;      // (narrow: the same in the warp)
            const uint32_t owner = static_cast<uint32_t>((owner_place << gs) | g);
            const uint32_t bar = lt_peer(bar_part, owner);
            const uint32_t dst = lt_peer(smem_u32(recv), owner) + static_cast<uint32_t>(place * row_chunks * kOwn + row - owner_place * kOwn) * 16u;
            for (int c = 0; c < pairs; c += 16) {              // the accumulator has 16, 32 or 64 columns
                uint32_t v[8], w[8];
                tmem_ld8(tmem_d2 + lane_base + static_cast<uint32_t>(mt * pairs_pad + c), v);
                tmem_ld8(tmem_d2 + lane_base + static_cast<uint32_t>(mt * pairs_pad + c + 8), w);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                constexpr uint32_t kFour = kOwn * 16u;
                const uint32_t at = dst + static_cast<uint32_t>(c >> 2) * kFour;
                lt_push16(at, bar, v[0], v[1], v[2], v[3]);
                if (c + 4 < pairs) lt_push16(at + kFour, bar, v[4], v[5], v[6], v[7]);
                if (c + 8 < pairs) lt_push16(at + 2 * kFour, bar, w[0], w[1], w[2], w[3]);
                if (c + 12 < pairs) lt_push16(at + 3 * kFour, bar, w[4], w[5], w[6], w[7]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");

    // ---- a warp (wide: a half-warp) owns four pairs and all owned columns: partial sums in a fixed order, so that the
    // result does not depend on timing, and (mean, M2) of the owned columns, pushed to every CTA
    if (kWide && pairs_pad == 16) {                            // the W_q slice, in the ring's place
        for (int mt = 0; mt < mtiles; ++mt)
            if (!mbar_wait(bar_d2 + 8u * mt, 0)) failed = 1;
        request_wq();
        cp_async_commit();
    }
    if (!mbar_wait(bar_part, 0)) failed = 1;
    constexpr int kIters = kWide ? 1 : 2, kPairLanes = kWide ? 4 : 8;
    const int first_lane = kWide ? lane & 16 : 0, sub_lane = lane - first_lane;
    const auto quad_at = [&](int it) { return kWide ? 2 * warp + (lane >> 4) : warp + 8 * it; };
    const auto quad_none = [&](int it) { return (kWide ? 2 * warp : warp + 8 * it) >= quads; };      // for the whole warp
    float x[kIters][kOwnPer][4];
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
        if (quad_none(it)) break;
        const int q = min(quad_at(it), quads - 1);
#pragma unroll
        for (int i = 0; i < kOwnPer; ++i) {
            const unsigned char* src = recv + static_cast<uint32_t>(q * kOwn + column + 16 * i) * 16u;
            const uint32_t sender = static_cast<uint32_t>(row_chunks * kOwn) * 16u;
            float4 part_sum[4];                                // senders of equal place modulo four (4, 8 or 16 of them)
#pragma unroll
            for (int k = 0; k < 4; ++k) part_sum[k] = *reinterpret_cast<const float4*>(src + static_cast<uint32_t>(k) * sender);
#pragma unroll
            for (int first = 4; first < (kWide ? 8 : 16); first += 4) {
                if (first >= senders) break;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 v = *reinterpret_cast<const float4*>(src + static_cast<uint32_t>(first + k) * sender);
                    part_sum[k].x += v.x; part_sum[k].y += v.y; part_sum[k].z += v.z; part_sum[k].w += v.w;
                }
            }
            x[it][i][0] = (part_sum[0].x + part_sum[1].x) + (part_sum[2].x + part_sum[3].x) + pre_bias[i];
            x[it][i][1] = (part_sum[0].y + part_sum[1].y) + (part_sum[2].y + part_sum[3].y) + pre_bias[i];
            x[it][i][2] = (part_sum[0].z + part_sum[1].z) + (part_sum[2].z + part_sum[3].z) + pre_bias[i];
            x[it][i][3] = (part_sum[0].w + part_sum[1].w) + (part_sum[2].w + part_sum[3].w) + pre_bias[i];
        }
        float2 moments;
        if constexpr (kWide) moments = lt_moments4(x[it]);
        else moments = lt_moments4(x[it][0]);
        const int pr = 4 * q + sub_lane / kPairLanes;
        if (pr < pairs && quad_at(it) < quads && sub_lane % kPairLanes == 0) stats_out[pr] = moments;
    }
    __syncthreads();
    // ... in messages of sixteen bytes (64 pairs: this exchange took 3 900 cycles with eight bytes a message)
    if (lane < (pairs + 1) >> 1) {                             // a lane two pairs, a warp two or one of the CTAs
        const float4 m = *reinterpret_cast<const float4*>(&stats_out[2 * lane]);
        const uint32_t at = smem_u32(&stats_in[rank * pairs_pad + 2 * lane]);
        for (uint32_t i = warp; i < static_cast<uint32_t>(C); i += kLtThreads / 32) {
            const uint32_t to = (i + rank) & static_cast<uint32_t>(C - 1);
            lt_push16(lt_peer(at, to), lt_peer(bar_stat, to), __float_as_uint(m.x), __float_as_uint(m.y), __float_as_uint(m.z), __float_as_uint(m.w));
        }
    }

    // ---- the pairs' statistics over the full width (equal counts: Chan's parallel variance), eight (four) lanes a pair, and
    // the normalised pairs [pair][kOwnStride] for the sequences' weighted sums
    float* own_y = reinterpret_cast<float*>(base + plan.own_y);
    if (!mbar_wait(bar_stat, 0)) failed = 1;
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
        if (quad_none(it)) break;
        const int q = min(quad_at(it), quads - 1);
        const int pr = min(4 * q + sub_lane / kPairLanes, pairs - 1), from = lane % kPairLanes;
        // sums of the means' distances from the first one, of their squares and of the M2, in the same exchanges
        const float pivot = stats_in[pr].x;
        float d1 = 0.0f, d2 = 0.0f, m2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 16 / kPairLanes; ++i)
            if (from + kPairLanes * i < C) {
                const float2 st = stats_in[(from + kPairLanes * i) * pairs_pad + pr];
                const float d = st.x - pivot;
                d1 += d;
                d2 = fmaf(d, d, d2);
                m2 += st.y;
            }
#pragma unroll
        for (int o = kPairLanes / 2; o > 0; o >>= 1) {
            d1 += __shfl_xor_sync(0xffffffffu, d1, o);
            d2 += __shfl_xor_sync(0xffffffffu, d2, o);
            m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        }
        const float mean = fmaf(d1, per, pivot);
        m2 = fmaf(static_cast<float>(kOwn), fmaxf(fmaf(-d1 * per, d1, d2), 0.0f), m2);
        const float rstd = rsqrtf(fmaf(m2, inv_d, a.eps));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float mj = __shfl_sync(0xffffffffu, mean, first_lane + kPairLanes * j), rj = __shfl_sync(0xffffffffu, rstd, first_lane + kPairLanes * j);
            if (4 * q + j < pairs && quad_at(it) < quads)
#pragma unroll
                for (int i = 0; i < kOwnPer; ++i)
                    own_y[(4 * q + j) * kOwnStride + column + 16 * i] = fmaf((x[it][i][j] - mj) * rj, pre_g[i], pre_bt[i]);
        }
    }
    __syncthreads();
    // every warp has read its accumulators: the tensor memory goes back now, off the kernel's exit path
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }

    // ---- context and residual update: column = lane (wide: and 32 + lane); the warps of a sequence share out the CTAs
    // that its updated columns are pushed to
    if (part < parts) {
#pragma unroll
        for (int i = 0; i < kResPer; ++i) {
            const int col = lane + 32 * i;
            if (col >= kOwn) continue;
            float ctx = 0.0f;
            for (int k0 = 0; k0 < K; k0 += 8) {
                float wk[8], y[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int at = my_seq * K + min(k0 + k, K - 1);
                    wk[k] = k0 + k < K ? weight_s[at] : 0.0f;
                    y[k] = own_y[at * kOwnStride + col];
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) ctx = wk[k] == 0.0f ? ctx : fmaf(wk[k], y[k], ctx);     // inactive slots contribute nothing
            }
            const float hval = bad_position ? pre_res[i] : fmaf(pre_mix, ctx, pre_res[i]);
            if (part == 0 && !bad_position) a.residual[static_cast<size_t>(s0 + my_seq) * D + own0 + col] = hval;
            const uint32_t at = smem_u32(&rows_in[my_seq * D + own0 + col]);
            for (uint32_t to_i = part; to_i < static_cast<uint32_t>(C); to_i += parts) {
                const uint32_t to = (to_i + rank) & static_cast<uint32_t>(C - 1);
                lt_push4(lt_peer(at, to), lt_peer(bar_rows, to), hval);
            }
        }
    }

    // ---- the next LayerNorm, of whole rows in every CTA: the warps of a sequence share its 128-column chunks
    cp_async_wait_all();                                       // this thread's pieces of the W_q slice
    if (!mbar_wait(bar_rows, 0)) failed = 1;
    __syncwarp();
    lt_cluster_arrive();                                       // nothing more is pushed to this CTA, nor by it
    unsigned char* rows16 = base + plan.rows;                  // [sequence][d] of 16 bits
    if (part < parts) {
        const float* row = rows_in + my_seq * D;
        // local moments of the lane's 4 row_tiles columns, then five exchanges of (mean, M2) of equal halves
        float4 h[kChunks128];
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < kChunks128; ++i) {
            h[i] = i < row_tiles ? *reinterpret_cast<const float4*>(row + 128 * i + 4 * lane) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            sum += (h[i].x + h[i].y) + (h[i].z + h[i].w);
        }
        float count = 4.0f * static_cast<float>(row_tiles), mean = sum * (1.0f / count), m2 = 0.0f;      
#pragma unroll
        for (int i = 0; i < kChunks128; ++i)
            if (i < row_tiles) {
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
        const float rstd = rsqrtf(fmaf(m2, inv_d, a.next_eps));
#pragma unroll
        for (int i = 0; i < kChunks128; ++i) {
            const int chunk = part + i * parts;
            if (chunk >= row_tiles) break;
            float4 v = h[0];
#pragma unroll
            for (int k = 1; k < kChunks128; ++k)
                if (chunk == k) v = h[k];
            const float4 g = next_g[i], b = next_b[i];
            const uint2 out = make_uint2(
                pack2(fmaf((v.x - mean) * rstd, g.x, b.x), fmaf((v.y - mean) * rstd, g.y, b.y), dtype),
                pack2(fmaf((v.z - mean) * rstd, g.z, b.z), fmaf((v.w - mean) * rstd, g.w, b.w), dtype));
            const int at = 128 * chunk + 4 * lane;
            *reinterpret_cast<uint2*>(rows16 + (my_seq * D + at) * 2) = out;
            if (at >= own0 && at < own0 + kOwn && !bad_position) {
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

int lt_validate(const LayerTailArgs& a, bool wide = false) {
    if (a.n_seq < 1 || a.k_out < 1 || a.k_out > kLtMaxPairs || a.max_t < 1) {
        set_error("relation_layer_tail: sizes must be positive and K at most 64");
        return RLM_ERR_SHAPE;
    }
    if (a.dtype != RLM_BF16 && a.dtype != RLM_F16) {
        set_error("relation_layer_tail: caches and weights must share bfloat16 or float16");
        return RLM_ERR_UNSUPPORTED;
    }
    if (a.hdim != 4 * a.d || (wide ? a.d != 768 : a.d != 128 && a.d != 256 && a.d != 512) || a.rdim < kBK || a.rdim % kBK != 0 || a.rdim > 256) {
        set_error(wide ? "relation_layer_tail_wide: needs H = 4 d with d = 768 and R a multiple of 64"
                       : "relation_layer_tail: needs H = 4 d with d in {128, 256, 512} and R a multiple of 64 up to 256");
        return RLM_ERR_UNSUPPORTED;
    }
    const int cluster = lt_cluster(a.d);
    if (a.query_weight && (a.n_query < cluster || a.n_query % (16 * cluster) != 0 || a.n_query / cluster > 64 || !a.query ||
                           static_cast<size_t>(a.n_query / cluster) * (a.d * 2 + 256) > static_cast<size_t>(a.rdim / kBK) * lt_hidden(a.d) * 128)) {
        set_error("relation_layer_tail: query projection width must be a multiple of 16 outputs per CTA (H / 128 CTAs), at most 64 each");
        return RLM_ERR_UNSUPPORTED;
    }
    // (a ring has to hold what takes its place: 64 pairs' partial sums are six tiles; in its last one the products' low parts)
    if (lt_smem_bytes(a.rdim, a.d, a.query_weight ? a.n_query / cluster : 0) > static_cast<uint32_t>(kSmemDynamicLimit) ||
        (lt_wide(a.d) && (lt_plan(a.rdim, a.d, true, kLtMaxPairs, 0).ring < 6 || a.rdim > 2 * kBK))) {
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

// The relation MLP of a whole-sequence pass in one kernel (sm_100a): gather, product, first layer, GELU,
// second layer, LayerNorm, softmax weights and weighted sum, with neither the hidden states nor the
// second layer's rows ever written to device memory.
//
//   hid[pair, h] = gelu( W_m[h, :] . (operand[a] * operand[p]) + expanded[a, h] + expanded[p, H + h] )
//   raw[pair, :] = W_2 hid[pair, :] + b_2
//   out[row, :]  = residual[row, :] + scale * sum_pairs u[pair] * LayerNorm(raw[pair, :])
//
// A row's pairs are its K partners (whole-sequence layer) or the K partners of each of its S anchor
// slots (multi-anchor layer, the slot weights folded into u).  Formulas: relation_hidden_cached and
// relation_norm_reduce (src/relation_lm/kernels/relation_reduce.py:72-146, 360-417 of the reference
// project) and the slot mixing of src/relation_lm/models/multi_relation_blocks.py:164-178.
//
// Why this shape.  As three kernels (hidden rows, GEMM, norm-reduce) the 16-bit hidden states make a
// round trip of 2 * pairs * H bytes each way: 1.07 GB written and read back for 262 144 pairs of
// H = 2048, beside a GELU epilogue that nothing overlaps.  Kept on chip, the second layer needs an
// fp32 accumulator of 128 pairs x d, all of an SM's tensor memory at d = 512; so a tile of 128 pairs
// belongs to C = 2 CTAs of a cluster (C = 1 for d <= 384): each accumulates d / C output columns and
// computes every C-th block of 64 hidden columns, which it passes on to the other through distributed
// shared memory (one bulk copy per 32 rows, completing on the receiver's mbarrier).
//
// kG = 2 pairs the tiles of two neighbouring CTAs on tcgen05.mma.cta_group::2 (256 pair rows, each CTA
// holding half of the weight rows): what bounds the kernel with kG = 1 is the stream of W_2 out of L2 —
// 2.5 MB of weights per 128 pairs — and pairing halves it.
//
// One CTA (24 warps), a persistent loop over tiles:
//   warps 0-15   epilogue: thread = pair row x 16 hidden columns per block; then the LayerNorm and
//                the weighted sum of the finished tile (thread = pair row x a quarter of the columns)
//   warps 16, 19 TMA producers of W_2 and of W_m tiles (apart: a full W_2 ring must not hold up W_m)
//   warps 17, 18 tcgen05.mma issue of the first and of the second layer (the first CTA of a pair; in the
//                second they forward its barriers to the first)
//   warps 20-23  gathers: operand products into the A tile of the next tile, and for every block the
//                expanded-cache segments of its pairs
// Pipelines: two hidden blocks per part in flight (one per epilogue group), two accumulators for the first
// layer, rings of gathered segments, W_m and W_2 tiles.  (Gathering into the hidden block that the epilogue
// then overwrites saved 16 KB per block, but put a gather's latency behind the second layer's last use of
// that block: 2 450 cycles per block of 64 hidden columns at three blocks in flight.)  Every wait is bounded; on expiry the kernel sets RLM_DEV_TIMEOUT, drains and returns.

#include <map>
#include <mutex>
#include <tuple>

#include "rlm_tcgen05.cuh"

namespace rlm {
namespace {

constexpr int kMlpEpiWarps = 16;
constexpr int kMlpGatherWarps = 4;
constexpr int kMlpThreads = 32 * (kMlpEpiWarps + 4 + kMlpGatherWarps);
constexpr int kMlpHC = 64;                       // hidden columns per block: one 128-byte swizzle atom of K
constexpr uint32_t kMlpBlock = kBM * 128u;       // a 128 x 64 16-bit block
constexpr uint32_t kMlpAncStride = 144;          // padded anchor-term row: conflict-free for rows of different anchors
constexpr int kMlpMaxStages = 4;
constexpr int kMlpHidden = 2;                    // hidden blocks in flight per part
constexpr int kMlpMaxTerms = 4;                  // gathered blocks in flight

struct MlpArgs {
    const void* expanded_cache;      // [B, T, 2H]
    const void* operand_cache;       // [B, T, R]
    const int32_t* anchor_index;     // [rows * S]
    const int32_t* partner_index;    // [rows * S, K]
    const float* scores;             // [rows * S, K]
    const uint8_t* active;           // [rows, S] or NULL
    const float* slot_weight;        // [S] or NULL
    const float* scale;              // one element or NULL (1)
    const float* second_bias;        // [d]
    const float* norm_w;             // [d]
    const float* norm_b;
    const float* residual;           // [rows out, d] or NULL
    float* out;                      // [rows out, d]
    int32_t* status;
    float eps;
    int slots, n_seq, rows_per_seq, max_t, rdim, hdim, d, k_shift, group_shift, limited;
    int n_pairs, n_tiles;            // tiles of 128 pairs
    int cols;                        // output columns per CTA (NC)
    int term_stages, w2_stages, wm_stages;
    uint32_t idesc1, idesc2;
};

// Shared-memory plan (byte offsets from the 1024-aligned dynamic base).
struct MlpPlan {
    uint32_t a, wm, w2, hid, term, anc, bias, gamma, beta, stats, u, prow, arow, total;
};

__host__ __device__ inline MlpPlan mlp_plan(int rdim, int cols, int outs, int group_ctas, int term_stages, int wm_stages,
                                            int w2_stages, int k_shift) {
    MlpPlan p;
    uint32_t off = 0;
    p.a = off;      off += static_cast<uint32_t>(rdim / kBK) * kMlpBlock;
    p.wm = off;     off += static_cast<uint32_t>(wm_stages * (rdim / kBK)) * (kMlpHC / group_ctas) * 128u;
    p.w2 = off;     off += static_cast<uint32_t>(w2_stages) * ((cols > 256 ? cols / 2 : cols) / group_ctas) * 128u;
    p.hid = off;    off += static_cast<uint32_t>(kMlpHidden * outs) * kMlpBlock;
    p.term = off;   off += static_cast<uint32_t>(term_stages) * kMlpBlock;
    p.anc = off;    off += static_cast<uint32_t>(term_stages) * (kBM >> k_shift) * kMlpAncStride;
    p.bias = off;   off += static_cast<uint32_t>(cols) * 4u;
    p.gamma = off;  off += static_cast<uint32_t>(cols) * 4u;
    p.beta = off;   off += static_cast<uint32_t>(cols) * 4u;
    p.stats = off;  off += static_cast<uint32_t>(4 * outs) * kBM * 8u;
    p.u = off;      off += 3u * kBM * 4u;
    p.prow = off;   off += 2u * kBM * 4u;
    p.arow = off;   off += 2u * (kBM >> k_shift) * 4u;
    p.total = off;
    return p;
}

struct MlpBars {
    unsigned long long a_full, a_empty, d2_full, d2_empty, stats_full;
    unsigned long long u_full[3], d1_full[2], d1_empty[2];
    unsigned long long wm_full[2], wm_empty[2], peer_wm[2];
    unsigned long long w2_full[kMlpMaxStages], w2_empty[kMlpMaxStages], peer_w2[kMlpMaxStages];
    unsigned long long hid_full[kMlpHidden][2], hid_empty[kMlpHidden];
    unsigned long long term_full[kMlpMaxTerms], term_empty[kMlpMaxTerms];
};

// ---- cluster primitives

__device__ __forceinline__ uint32_t mlp_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void mlp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t mlp_peer(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
__device__ __forceinline__ void mlp_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrivals at another CTA's barrier carry the default (CTA-scope) release: what they announce is tensor
// memory that has been read or shared memory that an async proxy wrote or will read (after
// fence.proxy.async), which mbarrier completion orders.  Values for another CTA travel by bulk copies and
// st.async, whose completion on the receiver's barrier makes them visible.
__device__ __forceinline__ void mlp_arrive_remote(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
__device__ __forceinline__ void mlp_expect_remote(uint32_t remote_bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(remote_bar), "r"(bytes) : "memory");
}
// Arrives at the pair leader's barrier at the same offset.
template <int kG>
__device__ __forceinline__ void mlp_arrive_leader(uint32_t bar, uint32_t leader) {
    if (kG == 1) mlp_arrive(bar);
    else mlp_arrive_remote(mlp_peer(bar, leader));
}
__device__ __forceinline__ void mlp_copy_cluster(uint32_t remote_dst, uint32_t src, uint32_t bytes, uint32_t remote_bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(remote_dst), "r"(src), "r"(bytes), "r"(remote_bar) : "memory");
}
// Stores two floats in another CTA and counts their 8 bytes on that CTA's barrier.
__device__ __forceinline__ void mlp_store_remote(uint32_t remote_dst, float x, float y, uint32_t remote_bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                 ::"r"(remote_dst), "f"(x), "f"(y), "r"(remote_bar) : "memory");
}
// Completes `bar` once this thread's cp.async copies so far have landed (one of its expected arrivals).
__device__ __forceinline__ void mlp_cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool kCluster>
__device__ __forceinline__ bool mlp_try_wait(uint32_t bar, uint32_t parity) {
    if (!kCluster) return mbar_try_wait(bar, parity);
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Once a wait of the CTA has expired no other one waits either, and a role whose wait
// returned false issues nothing any more: it only walks its loops to the end, so that the barriers that
// need all of its warps still meet.
template <bool kCluster = false>
__device__ __forceinline__ bool mlp_wait(uint32_t bar, uint32_t parity, volatile int* failed) {
    if (mlp_try_wait<kCluster>(bar, parity)) return true;
    const long long start = clock64();
    while (!*failed) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (mlp_try_wait<kCluster>(bar, parity)) return true;
        if (clock64() - start > (1ll << 31)) *failed = 1;
    }
    return false;
}
__device__ __forceinline__ void mlp_bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// ---- tcgen05 in either CTA group (a kernel uses one of them throughout)
//
// The issuing warps run their loops and waits with all lanes and predicate each tcgen05 instruction on one
// elected lane.  Inside an `if (lane == 0)` the compiler has to move every descriptor from vector to
// uniform registers one instruction at a time: 140 cycles per MMA, longer than a 128 x 64 x 16 MMA takes.

__device__ __forceinline__ bool mlp_elect() {
    uint32_t p;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(p));
    return p != 0;
}

template <int kG>
__device__ __forceinline__ void mlp_umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                         bool issue) {
    if (kG == 1)
        asm volatile(
            "{\n"
            ".reg .pred p, q;\n"
            "setp.ne.b32 p, %4, 0;\n"
            "setp.ne.b32 q, %5, 0;\n"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
            "}\n"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(issue)) : "memory");
    else
        asm volatile(
            "{\n"
            ".reg .pred p, q;\n"
            "setp.ne.b32 p, %4, 0;\n"
            "setp.ne.b32 q, %5, 0;\n"
            "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
            "}\n"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(issue)) : "memory");
}
// Arrives on the barrier at this offset in every CTA of `mask` when the MMAs issued so far are complete.
template <int kG>
__device__ __forceinline__ void mlp_commit(uint32_t bar, uint32_t mask, uint32_t self, bool issue) {
    const uint16_t m = static_cast<uint16_t>(mask);
    if (kG == 1 && mask == self)
        asm volatile(
            "{\n"
            ".reg .pred q;\n"
            "setp.ne.b32 q, %1, 0;\n"
            "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
            "}\n"
            ::"r"(bar), "r"(static_cast<uint32_t>(issue)) : "memory");
    else if (kG == 1)
        asm volatile(
            "{\n"
            ".reg .pred q;\n"
            "setp.ne.b32 q, %2, 0;\n"
            "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
            "}\n"
            ::"r"(bar), "h"(m), "r"(static_cast<uint32_t>(issue)) : "memory");
    else
        asm volatile(
            "{\n"
            ".reg .pred q;\n"
            "setp.ne.b32 q, %2, 0;\n"
            "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
            "}\n"
            ::"r"(bar), "h"(m), "r"(static_cast<uint32_t>(issue)) : "memory");
}

// Sums y[0 .. 16) over the 2^kLG lanes of a group, scattered: lane g of the group ends up with columns
// [g * (16 >> kLG), ...) in y[0 .. 16 >> kLG) (kLG = 5: both half-warps hold the same columns).
template <int kLG>
__device__ __forceinline__ void mlp_group_sum(float (&y)[16], int lane) {
    constexpr int kSteps = kLG > 4 ? 4 : kLG;
    if (kLG == 5)
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] += __shfl_xor_sync(0xffffffffu, y[k], 16);
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
        const int w = 8 >> s, bit = 1 << (kSteps - 1 - s);
        const bool upper = (lane & bit) != 0;
#pragma unroll
        for (int k = 0; k < w; ++k) {
            const float send = upper ? y[k] : y[k + w];
            const float keep = upper ? y[k + w] : y[k];
            y[k] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    }
}

// This warp's columns of a finished tile: the group's weighted sum of its rows, residual and store.
// `ur` = weight * rstd of this lane's row (0: the row contributes nothing, whatever it holds), `u_sum`, `ur_sum`,
// `urm_sum` = sums over the group of the weight, of ur and of ur * mean:
//   sum u LayerNorm(x + b) = gamma (sum ur x + b ur_sum - urm_sum) + beta u_sum.
// The next chunk's residual and tensor-memory columns are requested before a chunk is summed.
template <int kLG>
__device__ __forceinline__ void mlp_store_rows(uint32_t tmem, int cols, int lane, bool live, float ur, float u_sum, float ur_sum,
                                               float urm_sum, const float* bias, const float* gamma, const float* beta,
                                               const float* residual, float* out, uint32_t drained_bar, bool drained) {
    constexpr int kSteps = kLG > 4 ? 4 : kLG;
    constexpr int kCols = 16 >> kSteps;
    constexpr int kVec = kCols >= 4 ? 4 : kCols;
    const int c0 = (lane & ((1 << kSteps) - 1)) * kCols;
    const bool store = live && (kLG < 5 || lane < 16);
    float next[kCols];
#pragma unroll
    for (int k = 0; k < kCols; ++k) next[k] = 0.0f;
    const auto fetch = [&](int c) {
        if (!store || !residual) return;
#pragma unroll
        for (int k = 0; k < kCols; k += kVec) {
            if (kVec == 4) {
                const float4 r = *reinterpret_cast<const float4*>(residual + c + c0 + k);
                next[k] = r.x; next[k + 1 < kCols ? k + 1 : 0] = r.y; next[k + 2 < kCols ? k + 2 : 0] = r.z; next[k + 3 < kCols ? k + 3 : 0] = r.w;
            } else if (kVec == 2) {
                const float2 r = *reinterpret_cast<const float2*>(residual + c + c0 + k);
                next[k] = r.x; next[k + 1 < kCols ? k + 1 : 0] = r.y;
            } else {
                next[k] = residual[c + c0 + k];
            }
        }
    };
    fetch(0);
#pragma unroll 1
    for (int c = 0; c < cols; c += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + static_cast<uint32_t>(c), v);
        float res[kCols];
#pragma unroll
        for (int k = 0; k < kCols; ++k) res[k] = next[k];
        if (c + 16 < cols) fetch(c + 16);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c + 16 >= cols) {                            // the accumulator may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (drained) mlp_arrive_remote(drained_bar);
        }
        float y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = ur == 0.0f ? 0.0f : __uint_as_float(v[i]) * ur;
        mlp_group_sum<kLG>(y, lane);
        if (!store) continue;
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
            const int col = c + c0 + k;
            res[k] += fmaf(gamma[col], fmaf(bias[col], ur_sum, y[k] - urm_sum), beta[col] * u_sum);
        }
#pragma unroll
        for (int k = 0; k < kCols; k += kVec) {
            if (kVec == 4)
                *reinterpret_cast<float4*>(out + c + c0 + k) = make_float4(res[k], res[k + 1 < kCols ? k + 1 : 0], res[k + 2 < kCols ? k + 2 : 0], res[k + 3 < kCols ? k + 3 : 0]);
            else if (kVec == 2)
                *reinterpret_cast<float2*>(out + c + c0 + k) = make_float2(res[k], res[k + 1 < kCols ? k + 1 : 0]);
            else
                out[c + c0 + k] = res[k];
        }
    }
}

template <int kDt, int kG>
__global__ void __launch_bounds__(kMlpThreads, 1) relation_mlp_rows_kernel(
    const __grid_constant__ CUtensorMap map_wm, const __grid_constant__ CUtensorMap map_w2, const MlpArgs a, const int outs) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) MlpBars bars;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed_s;
    volatile int* failed = &failed_s;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // warp-uniform
    const int C = outs, R = a.rdim, H = a.hdim, NC = a.cols;
    const uint32_t rank = mlp_rank();
    const int o = static_cast<int>(rank) / kG, g = static_cast<int>(rank) % kG;      // output part, row group
    const uint32_t leader = static_cast<uint32_t>(o * kG);                           // issues the pair's MMAs
    const uint32_t pair_mask = ((1u << kG) - 1u) << leader;
    const int kblocks = R / kBK, J = H / (kMlpHC * C);
    const int cluster = static_cast<int>(blockIdx.x) / (C * kG), n_clusters = static_cast<int>(gridDim.x) / (C * kG);
    const int n_super = (a.n_tiles + kG - 1) / kG;

    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const MlpPlan plan = mlp_plan(R, NC, C, kG, a.term_stages, a.wm_stages, a.w2_stages, a.k_shift);
    const uint32_t s_a = smem_u32(base + plan.a), s_wm = smem_u32(base + plan.wm), s_w2 = smem_u32(base + plan.w2);
    const uint32_t s_hid = smem_u32(base + plan.hid);
    const uint32_t wm_kblock = (kMlpHC / kG) * 128u, wm_stage = static_cast<uint32_t>(kblocks) * wm_kblock;
    const int n_inst = NC > 256 ? 2 : 1, NI = NC / n_inst;
    const uint32_t w2_stage = static_cast<uint32_t>(NI / kG) * 128u;        // one instruction's weight rows
    float* bias_s = reinterpret_cast<float*>(base + plan.bias);
    float* gamma_s = reinterpret_cast<float*>(base + plan.gamma);
    float* beta_s = reinterpret_cast<float*>(base + plan.beta);
    float2* stats_s = reinterpret_cast<float2*>(base + plan.stats);
    float* u_s = reinterpret_cast<float*>(base + plan.u);

    if (tid == 0) {
        failed_s = 0;
        const auto init = [](unsigned long long* b, int count) { mbar_init(smem_u32(b), static_cast<uint32_t>(count)); };
        init(&bars.a_full, kMlpGatherWarps * kG);
        init(&bars.a_empty, 1);
        init(&bars.d2_full, 1);
        init(&bars.d2_empty, kMlpEpiWarps * kG);
        init(&bars.stats_full, C == 1 ? kMlpEpiWarps : 1);
        for (int i = 0; i < 3; ++i) init(&bars.u_full[i], kMlpGatherWarps);
        for (int i = 0; i < 2; ++i) {
            init(&bars.d1_full[i], 1);
            init(&bars.d1_empty[i], kMlpEpiWarps / 2 * kG);
            init(&bars.wm_full[i], 1);
            init(&bars.wm_empty[i], 1);
            init(&bars.peer_wm[i], 1);
        }
        for (int i = 0; i < kMlpMaxStages; ++i) {
            init(&bars.w2_full[i], 1);
            init(&bars.w2_empty[i], 1);
            init(&bars.peer_w2[i], 1);
        }
        for (int i = 0; i < kMlpHidden; ++i) {
            for (int b = 0; b < 2; ++b) init(&bars.hid_full[i][b], C == 1 ? kMlpEpiWarps / 2 : 4);
            init(&bars.hid_empty[i], C);
        }
        for (int i = 0; i < kMlpMaxTerms; ++i) {
            init(&bars.term_full[i], 32 * kMlpGatherWarps);
            init(&bars.term_empty[i], kMlpEpiWarps / 2);
        }
        fence_barrier_init();
    }
    if (warp == kMlpEpiWarps + 1) {
        if (kG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    for (int i = tid; i < NC; i += kMlpThreads) {       // parameters of this CTA's output columns
        bias_s[i] = a.second_bias[o * NC + i];
        gamma_s[i] = a.norm_w[o * NC + i];
        beta_s[i] = a.norm_b[o * NC + i];
    }
    griddep_sync();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    mlp_cluster_sync();                                  // every CTA's barriers are initialised
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d2 = __shfl_sync(0xffffffffu, tmem_slot, 0), tmem_d1 = tmem_d2 + static_cast<uint32_t>(NC);

    if (warp < kMlpEpiWarps) {
        // ------------------------------------------------------------ epilogue
        // Two groups of eight warps take the hidden blocks in turn, so that one group's waits and loads fall into
        // the other's arithmetic; thread = pair row x 32 of a block's 64 columns.
        const int row = 32 * (warp & 3) + lane, turn = warp >> 3, half = (warp >> 2) & 1;
        const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
        const uint32_t row_at = static_cast<uint32_t>((row >> 3) * 1024 + (row & 7) * 128);
        const unsigned char* anc = base + plan.anc + static_cast<uint32_t>(row >> a.k_shift) * kMlpAncStride + 64 * half;
        const uint32_t anc_stage = static_cast<uint32_t>(kBM >> a.k_shift) * kMlpAncStride;
        const int q = warp >> 2, quarter = NC / 4;                   // output columns of this warp in the last stage
        const int group = 1 << a.group_shift;
        const uint32_t d2_drained = mlp_peer(smem_u32(&bars.d2_empty), leader);
        int n = 0, ts = 0, tphase = 0, tix = 0, tix3 = 0, u_phase = 0;
        bool ok = true;
        for (int super = cluster; super < n_super; super += n_clusters, ++tix) {
            for (int j = 0; j < J; ++j, ++n) {
                const int slot = ts, phase = tphase, use = (n >> 1) & 1;
                if (++ts == a.term_stages) { ts = 0; tphase ^= 1; }
                if ((n & 1) != turn) continue;
                const unsigned char* term = base + plan.term + static_cast<uint32_t>(slot) * kMlpBlock + row_at;
                unsigned char* block = base + plan.hid + static_cast<uint32_t>(turn * C + o) * kMlpBlock;
                ok = ok && mlp_wait(smem_u32(&bars.d1_full[turn]), use, failed);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t v[2][16];
                tmem_ld16(tmem_d1 + lane_base + static_cast<uint32_t>(turn * kMlpHC + 32 * half), v[0]);
                tmem_ld16(tmem_d1 + lane_base + static_cast<uint32_t>(turn * kMlpHC + 32 * half + 16), v[1]);
                ok = ok && mlp_wait(smem_u32(&bars.term_full[slot]), phase, failed);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (ok && lane == 0) mlp_arrive_leader<kG>(smem_u32(&bars.d1_empty[turn]), leader);
                uint4 w[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float2 fa[4], fp[4];
                    unpack8_pairs(*reinterpret_cast<const uint4*>(anc + slot * anc_stage + 16 * c), kDt, fa);
                    unpack8_pairs(*reinterpret_cast<const uint4*>(term + ((static_cast<uint32_t>(4 * half + c) ^ (row & 7)) << 4)), kDt, fp);
                    uint32_t y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 acc = make_float2(__uint_as_float(v[c >> 1][8 * (c & 1) + 2 * i]),
                                                       __uint_as_float(v[c >> 1][8 * (c & 1) + 2 * i + 1]));
                        const float2 h = gelu_pair(__fadd2_rn(acc, __fadd2_rn(fa[i], fp[i])));
                        y[i] = pack2(h.x, h.y, kDt);
                    }
                    w[c] = make_uint4(y[0], y[1], y[2], y[3]);
                }
                __syncwarp();
                if (ok && lane == 0) mlp_arrive(smem_u32(&bars.term_empty[slot]));
                // the block's previous content has been consumed, here and where it was copied to
                ok = ok && mlp_wait(smem_u32(&bars.hid_empty[turn]), use ^ 1, failed);
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<uint4*>(block + row_at + ((static_cast<uint32_t>(4 * half + c) ^ (row & 7)) << 4)) = w[c];
                fence_proxy_async();                                  // the block -> tensor core, bulk copy
                const uint32_t full = smem_u32(&bars.hid_full[turn][o]);
                if (C == 1) {
                    __syncwarp();
                    if (ok && lane == 0) mlp_arrive(full);
                } else {
                    // both warps of these 32 rows have written their columns: 4 KB that are contiguous in the block
                    mlp_bar_sync(1 + 4 * turn + (warp & 3), 64);
                    if (ok && half == 0 && lane == 0) {
                        mlp_arrive(full);
                        const uint32_t part = smem_u32(block) + static_cast<uint32_t>(warp & 3) * 4096u;
                        for (int other = 0; other < C; ++other) {
                            if (other == o) continue;
                            const uint32_t to = static_cast<uint32_t>(other * kG + g);
                            const uint32_t bar = mlp_peer(full, to);
                            mlp_expect_remote(bar, 4096u);
                            mlp_copy_cluster(mlp_peer(part, to), part, 4096u, bar);
                        }
                    }
                }
            }
            // ---- the tile's second layer is complete: LayerNorm over d, weighted sum over the group
            const int tile = super * kG + g;
            const uint32_t tmem_row = tmem_d2 + lane_base + static_cast<uint32_t>(q * quarter);
            const float* bias = bias_s + q * quarter;
            ok = ok && mlp_wait(smem_u32(&bars.d2_full), tix & 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (C > 1 && ok && tid == 0) mbar_expect_tx(smem_u32(&bars.stats_full), static_cast<uint32_t>(4 * C * kBM * 8));
            // statistics of this thread's columns about the mean of the first sixteen: one pass over the accumulator
            float shift = 0.0f, s1 = 0.0f, s2 = 0.0f;
#pragma unroll 1
            for (int c = 0; c < quarter; c += 16) {
                uint32_t v[16];
                tmem_ld16(tmem_row + static_cast<uint32_t>(c), v);
                float x[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 b = *reinterpret_cast<const float4*>(bias + c + 4 * i);
                    x[4 * i] = b.x; x[4 * i + 1] = b.y; x[4 * i + 2] = b.z; x[4 * i + 3] = b.w;
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c == 0) {
                    float sum = 0.0f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum += __uint_as_float(v[i]) + x[i];
                    shift = sum * 0.0625f;
                }
                float t1 = 0.0f, t2 = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float y = (__uint_as_float(v[i]) + x[i]) - shift;
                    t1 += y;
                    t2 = fmaf(y, y, t2);
                }
                s1 += t1;
                s2 += t2;
            }
            const float inv_quarter = 1.0f / static_cast<float>(quarter);
            const float mean_q = fmaf(s1, inv_quarter, shift), m2 = fmaf(-s1 * inv_quarter, s1, s2);
            // every CTA of the tile receives (mean, sum of squares) of all quarters
            float2* mine = stats_s + (o * 4 + q) * kBM + row;
            if (C == 1) {
                *mine = make_float2(mean_q, m2);
                __syncwarp();
                if (ok && lane == 0) mlp_arrive(smem_u32(&bars.stats_full));
                ok = ok && mlp_wait(smem_u32(&bars.stats_full), tix & 1, failed);
            } else {
                for (int other = 0; ok && other < C; ++other) {
                    const uint32_t to = static_cast<uint32_t>(other * kG + g);
                    mlp_store_remote(mlp_peer(smem_u32(mine), to), mean_q, m2, mlp_peer(smem_u32(&bars.stats_full), to));
                }
                ok = ok && mlp_wait<true>(smem_u32(&bars.stats_full), tix & 1, failed);
            }
            float mean = 0.0f, total = 0.0f;
            for (int i = 0; i < 4 * C; ++i) mean += stats_s[i * kBM + row].x;
            mean *= C == 1 ? 0.25f : 0.125f;
            for (int i = 0; i < 4 * C; ++i) {
                const float2 s = stats_s[i * kBM + row];
                total += fmaf(static_cast<float>(quarter) * (s.x - mean), s.x - mean, s.y);
            }
            const float rstd = rsqrtf(total / static_cast<float>(a.d) + a.eps);
            ok = ok && mlp_wait(smem_u32(&bars.u_full[tix3]), u_phase, failed);
            const float u = u_s[tix3 * kBM + row];
            if (++tix3 == 3) { tix3 = 0; u_phase ^= 1; }
            const float ur = u == 0.0f ? 0.0f : u * rstd;
            float u_sum = u, ur_sum = ur, urm_sum = u == 0.0f ? 0.0f : ur * mean;
            for (int s = 1; s < group; s <<= 1) {
                u_sum += __shfl_xor_sync(0xffffffffu, u_sum, s);
                ur_sum += __shfl_xor_sync(0xffffffffu, ur_sum, s);
                urm_sum += __shfl_xor_sync(0xffffffffu, urm_sum, s);
            }
            const int pair = tile * kBM + row;
            const bool live = ok && pair < a.n_pairs;
            const size_t at = (live ? static_cast<size_t>(pair >> a.group_shift) : 0) * a.d + static_cast<size_t>(o * NC + q * quarter);
            const float* res = a.residual ? a.residual + at : nullptr;
            const float *gm = gamma_s + q * quarter, *bt = beta_s + q * quarter;
            float* out = a.out + at;
            const bool drained = ok && lane == 0;
#define MLP_STORE(kLG) mlp_store_rows<kLG>(tmem_row, quarter, lane, live, ur, u_sum, ur_sum, urm_sum, bias, gm, bt, res, out, d2_drained, drained)
            switch (a.group_shift) {
                case 1: MLP_STORE(1); break;
                case 2: MLP_STORE(2); break;
                case 3: MLP_STORE(3); break;
                case 4: MLP_STORE(4); break;
                default: MLP_STORE(5); break;
            }
#undef MLP_STORE
        }
    } else if (warp == kMlpEpiWarps) {
        // ------------------------------------------------------------ W_2 tiles
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w2) : "memory");
            int ws = 0, wphase = 0;
            bool ok = true;
            for (int super = cluster; ok && super < n_super; super += n_clusters)
                for (int j = 0; ok && j < J; ++j)
                    for (int part = 0; part < C; ++part)
                        for (int i = 0; i < n_inst; ++i) {
                            const int b = part == 0 ? o : 1 - o;
                            const uint32_t bar = smem_u32(&bars.w2_full[ws]);
                            ok = ok && mlp_wait(smem_u32(&bars.w2_empty[ws]), wphase ^ 1, failed);
                            if (!ok) break;
                            mbar_expect_tx(bar, w2_stage);
                            tma_load_2d(s_w2 + ws * w2_stage, &map_w2, (j * C + b) * kMlpHC, o * NC + i * NI + g * (NI / kG), bar);
                            if (++ws == a.w2_stages) { ws = 0; wphase ^= 1; }
                        }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 3) {
        // ------------------------------------------------------------ W_m tiles
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_wm) : "memory");
            int ms = 0, mphase = 0;
            bool ok = true;
            for (int super = cluster; ok && super < n_super; super += n_clusters)
                for (int j = 0; j < J; ++j) {
                    const uint32_t bar = smem_u32(&bars.wm_full[ms]);
                    ok = ok && mlp_wait(smem_u32(&bars.wm_empty[ms]), mphase ^ 1, failed);
                    if (!ok) break;
                    mbar_expect_tx(bar, wm_stage);
                    for (int kb = 0; kb < kblocks; ++kb)
                        tma_load_2d(s_wm + ms * wm_stage + kb * wm_kblock, &map_wm, kb * kBK,
                                    (j * C + o) * kMlpHC + g * (kMlpHC / kG), bar);
                    if (++ms == a.wm_stages) { ms = 0; mphase ^= 1; }
                }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 1) {
        // ------------------------------------------------------------ first layer: D1[n & 1] = products x W_m block
        const bool elected = mlp_elect(), issue = g == 0;
        const uint64_t a_desc = smem_desc_sw128(s_a), w_desc = smem_desc_sw128(s_wm);
        int ms = 0, mphase = 0, p = 0, tix = 0;
        bool ok = true;
        for (int super = cluster; ok && super < n_super; super += n_clusters, ++tix) {
            if (issue) ok = ok && mlp_wait(smem_u32(&bars.a_full), tix & 1, failed);
            for (int j = 0; ok && j < J; ++j, ++p) {
                ok = ok && mlp_wait(smem_u32(&bars.wm_full[ms]), mphase, failed);
                if (issue) {
                    if (kG == 2) ok = ok && mlp_wait(smem_u32(&bars.peer_wm[ms]), mphase, failed);
                    ok = ok && mlp_wait(smem_u32(&bars.d1_empty[p & 1]), ((p >> 1) & 1) ^ 1, failed);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const bool go = elected && ok;
                    const uint32_t d_at = tmem_d1 + static_cast<uint32_t>((p & 1) * kMlpHC);
                    const uint64_t wd = w_desc + (static_cast<uint32_t>(ms) * wm_stage >> 4);
#pragma unroll 2
                    for (int kb = 0; kb < kblocks; ++kb)
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; ++kk)
                            mlp_umma<kG>(d_at, a_desc + kb * (kMlpBlock >> 4) + 2 * kk, wd + kb * (wm_kblock >> 4) + 2 * kk, a.idesc1,
                                         (kb > 0 || kk > 0) ? 1u : 0u, go);
                    mlp_commit<kG>(smem_u32(&bars.d1_full[p & 1]), pair_mask, pair_mask, go);
                    mlp_commit<kG>(smem_u32(&bars.wm_empty[ms]), pair_mask, pair_mask, go);
                    if (j + 1 == J) mlp_commit<kG>(smem_u32(&bars.a_empty), pair_mask, pair_mask, go);
                } else if (ok && elected) {
                    mlp_arrive_remote(mlp_peer(smem_u32(&bars.peer_wm[ms]), leader));
                }
                if (++ms == a.wm_stages) { ms = 0; mphase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 2) {
        // ------------------------------------------------------------ second layer: D2 += hidden blocks x W_2 columns
        const bool elected = mlp_elect(), issue = g == 0;
        const uint64_t h_desc = smem_desc_sw128(s_hid), w_desc = smem_desc_sw128(s_w2);
        int ws = 0, wphase = 0, n = 0, tix = 0;
        bool ok = true;
        for (int super = cluster; ok && super < n_super; super += n_clusters, ++tix) {
            if (issue) ok = ok && mlp_wait(smem_u32(&bars.d2_empty), (tix & 1) ^ 1, failed);
            for (int j = 0; ok && j < J; ++j, ++n) {
                const int d = n & 1;
                for (int part = 0; part < C; ++part) {
                    const int b = part == 0 ? o : 1 - o;          // this CTA's own block first: the other one is still on its way
                    ok = ok && mlp_wait(smem_u32(&bars.hid_full[d][b]), (n >> 1) & 1, failed);
                    const uint64_t hd = h_desc + (static_cast<uint32_t>(d * C + b) * kMlpBlock >> 4);
                    for (int i = 0; i < n_inst; ++i) {
                        ok = ok && mlp_wait(smem_u32(&bars.w2_full[ws]), wphase, failed);
                        if (issue) {
                            if (kG == 2) ok = ok && mlp_wait(smem_u32(&bars.peer_w2[ws]), wphase, failed);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const bool go = elected && ok;
                            const uint64_t wd = w_desc + (static_cast<uint32_t>(ws) * w2_stage >> 4);
#pragma unroll
                            for (int kk = 0; kk < kBK / 16; ++kk)
                                mlp_umma<kG>(tmem_d2 + static_cast<uint32_t>(i * NI), hd + 2 * kk, wd + 2 * kk, a.idesc2,
                                             (j > 0 || part > 0 || kk > 0) ? 1u : 0u, go);
                            mlp_commit<kG>(smem_u32(&bars.w2_empty[ws]), pair_mask, pair_mask, go);
                            if (i + 1 == n_inst)
                                mlp_commit<kG>(smem_u32(&bars.hid_empty[d]), ((1u << kG) - 1u) << (b * kG), pair_mask, go);
                        } else if (ok && elected) {
                            // this CTA's hidden block and weight rows are there
                            mlp_arrive_remote(mlp_peer(smem_u32(&bars.peer_w2[ws]), leader));
                        }
                        if (++ws == a.w2_stages) { ws = 0; wphase ^= 1; }
                    }
                }
                if (issue && j + 1 == J) mlp_commit<kG>(smem_u32(&bars.d2_full), pair_mask, pair_mask, elected && ok);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ gathers
        const int gt = tid - 32 * (kMlpEpiWarps + 4), gw = gt >> 5;
        int* prow_s = reinterpret_cast<int*>(base + plan.prow);
        int* arow_s = reinterpret_cast<int*>(base + plan.arow);
        const int K = 1 << a.k_shift, anchors = kBM >> a.k_shift, chunks = R / 8, rows_per_warp = 32 / chunks;
        const size_t op_row = static_cast<size_t>(R) * 2, ex_row = static_cast<size_t>(H) * 4;
        const char* operand = static_cast<const char*>(a.operand_cache);
        const char* expanded = static_cast<const char*>(a.expanded_cache);
        const int cc = lane % chunks, r_first = gw * rows_per_warp + lane / chunks, r_step = kMlpGatherWarps * rows_per_warp;
        int ts = 0, tphase = 0, tix = 0, u_at = 0;
        bool ok = true;
        // This thread's pair of tile `super`: cache rows of its partner and anchor into buffer `b`, its weight into u.
        const auto indices = [&](int super, int b) {
            const int pair = (super * kG + g) * kBM + gt;
            int prow = -1, arow = -1;
            float u = 0.0f;
            if (pair < a.n_pairs) {
                const int srow = pair >> a.k_shift, k = pair & (K - 1);
                const int query = srow / a.slots, slot = srow - query * a.slots;
                const int seq = query / a.rows_per_seq, t = query - seq * a.rows_per_seq;
                prow = seq * a.max_t + min(max(a.partner_index[pair], 0), a.max_t - 1);
                arow = seq * a.max_t + min(max(a.anchor_index[srow], 0), a.max_t - 1);
                int k_limit = K;
                if (a.limited) k_limit = min(max(32 - __clz(t + 1), 1), K);          // ceil(log2(t + 2))
                const float* sc = a.scores + (static_cast<size_t>(srow) << a.k_shift);
                float mx = -1.0e4f, mine = kNegInf, den = 0.0f;
                for (int i = 0; i < K; ++i)
                    if (i < k_limit && sc[i] > -1.0e30f) {
                        mx = fmaxf(mx, sc[i]);
                        if (i == k) mine = sc[i];
                    }
                for (int i = 0; i < K; ++i)
                    if (i < k_limit && sc[i] > -1.0e30f) den += expf(sc[i] - mx);
                u = mine > -1.0e30f ? expf(mine - mx) / fmaxf(den, 1.0e-9f) : 0.0f;
                if (a.slot_weight) {
                    float all = 0.0f, own = 0.0f;
                    for (int s = 0; s < a.slots; ++s) {
                        const float w = a.active[static_cast<size_t>(query) * a.slots + s] ? a.slot_weight[s] : 0.0f;
                        all += w;
                        if (s == slot) own = w;
                    }
                    u *= own / fmaxf(all, 1.0e-9f);
                }
                if (a.scale) u *= *a.scale;
            }
            prow_s[b * kBM + gt] = prow;
            if ((gt & (K - 1)) == 0) arow_s[b * anchors + (gt >> a.k_shift)] = arow;
            u_s[u_at * kBM + gt] = u;
            __syncwarp();
            if (ok && lane == 0) mlp_arrive(smem_u32(&bars.u_full[u_at]));
            if (++u_at == 3) u_at = 0;
        };
        indices(cluster, 0);
        for (int super = cluster; super < n_super; super += n_clusters, ++tix) {
            const int* prow_t = prow_s + (tix & 1) * kBM;
            const int* arow_t = arow_s + (tix & 1) * anchors;
            mlp_bar_sync(9, 32 * kMlpGatherWarps);           // this tile's rows are written, the other buffer is no longer read
            // A tile: products of the operand rows, a lane per 16-byte chunk, eight rows' loads in flight
            ok = ok && mlp_wait(smem_u32(&bars.a_empty), (tix & 1) ^ 1, failed);
            for (int r0 = r_first; r0 < kBM; r0 += 8 * r_step) {
                uint4 pv[8], av[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = r0 + i * r_step, prow = r < kBM ? prow_t[r] : -1;
                    pv[i] = av[i] = make_uint4(0, 0, 0, 0);
                    if (prow >= 0) {
                        pv[i] = *reinterpret_cast<const uint4*>(operand + prow * op_row + 16 * cc);
                        av[i] = *reinterpret_cast<const uint4*>(operand + arow_t[r >> a.k_shift] * op_row + 16 * cc);
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = r0 + i * r_step;
                    if (r >= kBM) break;
                    float fp[8], fa[8];
                    unpack8(pv[i], kDt, fp);
                    unpack8(av[i], kDt, fa);
                    *reinterpret_cast<uint4*>(base + plan.a + swizzled(r, cc, kMlpBlock)) =
                        make_uint4(pack2(fp[0] * fa[0], fp[1] * fa[1], kDt), pack2(fp[2] * fa[2], fp[3] * fa[3], kDt),
                                   pack2(fp[4] * fa[4], fp[5] * fa[5], kDt), pack2(fp[6] * fa[6], fp[7] * fa[7], kDt));
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (ok && lane == 0) mlp_arrive_leader<kG>(smem_u32(&bars.a_full), leader);
            // the expanded-cache segments of every block of this CTA
            const int c = gt & 7;
            int rows[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) rows[i] = prow_t[(gt >> 3) + 16 * i];
            for (int j = 0; j < J; ++j) {
                const size_t h_bytes = static_cast<size_t>((j * C + o) * kMlpHC) * 2 + 16 * c;
                const uint32_t block = smem_u32(base + plan.term) + static_cast<uint32_t>(ts) * kMlpBlock;
                ok = ok && mlp_wait(smem_u32(&bars.term_empty[ts]), tphase ^ 1, failed);
                if (ok) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (rows[i] >= 0)
                            cp_async16(block + swizzled((gt >> 3) + 16 * i, c, kMlpBlock),
                                       expanded + rows[i] * ex_row + static_cast<size_t>(H) * 2 + h_bytes);
                    for (int r = gt >> 3; r < anchors; r += 16) {
                        const int arow = arow_t[r];
                        if (arow >= 0)
                            cp_async16(smem_u32(base + plan.anc) + static_cast<uint32_t>(ts * anchors + r) * kMlpAncStride + 16 * c,
                                       expanded + arow * ex_row + h_bytes);
                    }
                    mlp_cp_async_arrive(smem_u32(&bars.term_full[ts]));
                }
                if (++ts == a.term_stages) { ts = 0; tphase ^= 1; }
                if (j == 0 && super + n_clusters < n_super) indices(super + n_clusters, (tix & 1) ^ 1);
            }
        }
        cp_async_wait_all();
    }
    // ---- leave together: no CTA may go while another still reads or signals its shared memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    mlp_cluster_sync();
    if (tid == 0 && failed_s && a.status) atomicOr(a.status, RLM_DEV_TIMEOUT);
    if (warp == kMlpEpiWarps + 1) {
        if (kG == 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_d2) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_d2) : "memory");
    }
}

// ------------------------------------------------------------------ host

struct MlpShape { int outs, cols, term_stages, wm_stages, w2_stages; uint32_t smem; bool ok; };

bool power_of_two(int v) { return v > 0 && (v & (v - 1)) == 0; }

int log2_of(int v) {
    int s = 0;
    while ((1 << s) < v) ++s;
    return s;
}

// Output columns per CTA (tensor memory: cols of the second layer + 128 of the first), and the deepest
// pipelines that fit the shared memory: three gathered blocks first (a gather is an L2 or DRAM round trip),
// then W_2 stages.
MlpShape mlp_shape(int rdim, int hdim, int d, int k_shift, int group_ctas) {
    MlpShape s{};
    s.outs = d <= 384 ? 1 : 2;
    s.cols = d / s.outs;
    if (d % s.outs != 0 || s.cols % 64 != 0 || s.cols > 384 || hdim % (kMlpHC * s.outs) != 0) return s;
    for (int terms = 3; terms >= 2; --terms)
        for (int wm = 2; wm >= 1; --wm)
            for (int w2 = kMlpMaxStages; w2 >= 3 - (terms == 2); --w2) {
                const MlpPlan p = mlp_plan(rdim, s.cols, s.outs, group_ctas, terms, wm, w2, k_shift);
                if (p.total + 1024 <= static_cast<uint32_t>(kSmemDynamicLimit)) {
                    s.term_stages = terms;
                    s.w2_stages = w2;
                    s.wm_stages = wm;
                    s.smem = p.total + 1024;
                    s.ok = true;
                    return s;
                }
            }
    return s;
}

constexpr int kGroupCtas = 2;

// Clusters of this kernel that the device runs at a time (asked once per kernel, size and device): the grid
// is persistent, a cluster beyond that number would only start when another has finished all its tiles.
int mlp_clusters(const void* kernel, int cluster, uint32_t smem) {
    static std::mutex mutex;
    static std::map<std::tuple<const void*, int, uint32_t, int>, int> known;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) cudaGetLastError();
    std::lock_guard<std::mutex> lock(mutex);
    int& n = known[std::make_tuple(kernel, cluster, smem, device)];
    if (n == 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(static_cast<unsigned>(cluster));
        config.blockDim = dim3(kMlpThreads);
        config.dynamicSmemBytes = smem;
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = static_cast<unsigned>(cluster);
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &config) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sm_count() / cluster;
        }
    }
    return n;
}

template <int kDt, int kG>
int launch_mlp(const MlpArgs& a0, const MlpShape& s, const void* product_weight, const void* second_weight, void* stream) {
    MlpArgs a = a0;
    CUtensorMap map_wm, map_w2;
    const int n_inst = s.cols > 256 ? 2 : 1;
    if (!make_map(&map_wm, product_weight, a.hdim, a.rdim, a.rdim, kMlpHC / kG, kDt) ||
        !make_map(&map_w2, second_weight, a.d, a.hdim, a.hdim, s.cols / n_inst / kG, kDt)) {
        set_error("relation_mlp_rows: tensor map encoding failed");
        return RLM_ERR_LAUNCH;
    }
    auto* kernel = relation_mlp_rows_kernel<kDt, kG>;
    if (int rc = allow_large_smem(reinterpret_cast<const void*>(kernel), kSmemPerCta)) return rc;
    const int cluster = s.outs * kG, n_super = (a.n_tiles + kG - 1) / kG;
    const int most = mlp_clusters(reinterpret_cast<const void*>(kernel), cluster, s.smem);
    const int clusters = n_super < most ? n_super : most;
    launch_kernel_cluster(kernel, dim3(clusters * cluster), dim3(kMlpThreads), static_cast<unsigned>(cluster), s.smem, stream,
                          map_wm, map_w2, a, s.outs);
    count_launch();
    return check_launch("relation_mlp_rows_kernel");
}
}  // namespace
}  // namespace rlm

extern "C" int rlm_relation_mlp_rows_supported(int k_out, int slots, int relation_dim, int hidden_dim, int d_model, int dtype) {
    using namespace rlm;
    if (dtype != RLM_BF16 && dtype != RLM_F16) return 0;
    if (!power_of_two(k_out) || !power_of_two(slots) || k_out * slots > 32 || k_out < 2 || slots > 8) return 0;
    if (relation_dim != 64 && relation_dim != 128) return 0;
    if (d_model < 64 || hidden_dim < kMlpHC) return 0;
    return mlp_shape(relation_dim, hidden_dim, d_model, log2_of(k_out), kGroupCtas).ok ? 1 : 0;
}

extern "C" int rlm_relation_mlp_rows(
    const void* expanded_cache, const void* operand_cache, const int32_t* anchor_index, const int32_t* partner_index,
    const float* partner_scores, const uint8_t* anchor_active, const float* slot_weight, const float* scale,
    const void* product_weight, const void* second_weight, const float* second_bias, const float* norm_weight,
    const float* norm_bias, float norm_eps, const float* residual, float* out, int n_rows, int slots, int n_seq,
    int rows_per_seq, int max_t, int relation_dim, int hidden_dim, int d_model, int k_out, int limit_by_position, int dtype,
    int32_t* status, void* stream) {
    using namespace rlm;
    if (n_rows == 0) return RLM_OK;
    const void* need[] = {expanded_cache, operand_cache, anchor_index, partner_index, partner_scores, product_weight,
                          second_weight, second_bias, norm_weight, norm_bias, out};
    for (const void* q : need)
        if (!q) { set_error("relation_mlp_rows: NULL pointer"); return RLM_ERR_NULL; }
    if ((slot_weight != nullptr) != (anchor_active != nullptr)) {
        set_error("relation_mlp_rows: slot weights and anchor activity come together");
        return RLM_ERR_NULL;
    }
    if (!rlm_relation_mlp_rows_supported(k_out, slots, relation_dim, hidden_dim, d_model, dtype)) {
        set_error("relation_mlp_rows: sizes outside this kernel's range");
        return RLM_ERR_UNSUPPORTED;
    }
    if (n_rows < 0 || n_seq < 1 || rows_per_seq < 1 || max_t < 1 || static_cast<int64_t>(n_seq) * rows_per_seq < n_rows ||
        static_cast<int64_t>(n_rows) * slots * k_out > 0x7fffffff - 2 * kBM || static_cast<int64_t>(n_seq) * max_t > 0x7fffffff) {
        set_error("relation_mlp_rows: inconsistent sizes");
        return RLM_ERR_SHAPE;
    }
    for (const void* q : {expanded_cache, operand_cache, product_weight, second_weight, static_cast<const void*>(out),
                          static_cast<const void*>(residual)})
        if (!aligned16(q)) { set_error("relation_mlp_rows: tensors must be 16-byte aligned"); return RLM_ERR_ALIGN; }
    const int k_shift = log2_of(k_out);
    const MlpShape s = mlp_shape(relation_dim, hidden_dim, d_model, k_shift, kGroupCtas);
    const int n_inst = s.cols > 256 ? 2 : 1;
    const uint32_t fmt = dtype == RLM_BF16 ? 1u : 0u;
    const auto idesc = [&](int n) {
        return (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
               (static_cast<uint32_t>((kBM * kGroupCtas) >> 4) << 24);
    };
    MlpArgs a{};
    a.expanded_cache = expanded_cache;
    a.operand_cache = operand_cache;
    a.anchor_index = anchor_index;
    a.partner_index = partner_index;
    a.scores = partner_scores;
    a.active = anchor_active;
    a.slot_weight = slot_weight;
    a.scale = scale;
    a.second_bias = second_bias;
    a.norm_w = norm_weight;
    a.norm_b = norm_bias;
    a.residual = residual;
    a.out = out;
    a.status = status;
    a.eps = norm_eps;
    a.slots = slots;
    a.n_seq = n_seq;
    a.rows_per_seq = rows_per_seq;
    a.max_t = max_t;
    a.rdim = relation_dim;
    a.hdim = hidden_dim;
    a.d = d_model;
    a.k_shift = k_shift;
    a.group_shift = log2_of(k_out * slots);
    a.limited = limit_by_position ? 1 : 0;
    a.n_pairs = n_rows * slots * k_out;
    a.n_tiles = (a.n_pairs + kBM - 1) / kBM;
    a.cols = s.cols;
    a.term_stages = s.term_stages;
    a.w2_stages = s.w2_stages;
    a.wm_stages = s.wm_stages;
    a.idesc1 = idesc(kMlpHC);
    a.idesc2 = idesc(s.cols / n_inst);
    return dtype == RLM_BF16 ? launch_mlp<RLM_BF16, kGroupCtas>(a, s, product_weight, second_weight, stream)
                             : launch_mlp<RLM_F16, kGroupCtas>(a, s, product_weight, second_weight, stream);
}

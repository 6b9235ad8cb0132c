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
// belongs to C = 2 CTAs of a cluster (C = 1 for d <= 384 and more than 33 pairs of tiles): each accumulates d / C output columns and
// computes every C-th block of 64 hidden columns, which it passes on to the other through distributed
// shared memory (one bulk copy per 32 rows, completing on the receiver's mbarrier).
//
// The tiles of two neighbouring CTAs are paired on tcgen05.mma.cta_group::2 (256 pair rows, each CTA holding
// half of the weight rows): every 128 pairs otherwise stream 2.5 MB of weights out of L2, more than its
// bandwidth allows at the tensor cores' rate; pairing halves it.
//
// The expanded-cache terms join the first layer's accumulator as matrix products, so that the epilogue is GELU
// and nothing else: the partners' segments, gathered as a 128 x 64 block in operand layout, times the identity,
// and the anchors' segments selected by a one-hot matrix.  Both are exact in the fp32 accumulator.  (Added
// in the epilogue instead they cost a third of its instructions, and the epilogue was the bound.)  An infinity or NaN
// in an anchor's segment would reach every row of the product (zero times infinity), so the gathering threads look at
// what they place: such a chunk enters as zeros, and its anchor is marked for the epilogue, which makes the rows
// that selected it NaN.  (A partner's segment only meets its own row.)
//
// One CTA (32 warps, registers shifted to the epilogue by setmaxnreg), a persistent loop over tiles:
//   warps 0-15   epilogue: thread = pair row x 32 columns of a hidden block; then the LayerNorm and the
//                weighted sum of the finished tile (thread = pair row x a quarter of the columns)
//   warps 16, 17 TMA producers of W_2 and of W_m tiles (apart: a full W_2 ring must not hold up W_m)
//   warps 18, 19 tcgen05.mma issue of the first and of the second layer (the first CTA of a pair; in the
//                second they forward its barriers to the first)
//   warps 20-23  gathers of the expanded-cache segments (the partners' by cp.async, the anchors' through registers; as
//                TMA row gathers, tile::gather4, a block of 128 + 32 rows took 3 500 cycles instead of 1 000)
//   warps 24-31  indices, weights u, and the operand products of the next tile (the A tile): in registers
//                while the current tile runs, into shared memory the moment its last product is done
// Hidden columns go in units of 128 (two blocks of 64, one per epilogue group): up to 256 output columns per
// CTA leave tensor memory for two units of the first layer's accumulator, more for one, which is then
// handed over block by block.  Every wait is bounded; on expiry the kernel sets RLM_DEV_TIMEOUT, drains
// and returns.

#include <map>
#include <mutex>
#include <tuple>

#include "rlm_tcgen05.cuh"

namespace rlm {
namespace {

constexpr int kMlpEpiWarps = 16;
constexpr int kMlpGatherWarps = 4;
constexpr int kMlpOperandWarps = 8;
constexpr int kMlpThreads = 32 * (kMlpEpiWarps + 4 + kMlpGatherWarps + kMlpOperandWarps);
// Registers per thread by warpgroup after start-up; launched with 64 each, 8 warpgroups: 4 * 80 + 2 * 40 + 2 * 56 = 8 * 64.
constexpr int kMlpEpiRegs = 80, kMlpIssueRegs = 40, kMlpOperandRegs = 56;
constexpr int kG = 2;                            // CTAs whose MMAs are paired
constexpr int kMlpHC = 64;                       // hidden columns per block: one 128-byte swizzle atom of K
constexpr uint32_t kMlpBlock = kBM * 128u;       // a 128 x 64 16-bit block
constexpr int kMlpMaxStages = 4;
constexpr int kMlpHidden = 2;                    // hidden blocks in flight per part
constexpr int kMlpMaxTerms = 4;                  // gathered blocks in flight
// Tiles whose marks (anchors that are not finite) have slots of their own.  A slot is cleared with the rows of the tile
// before its next one, a moment that knows the epilogue only to be past the tile five before: the first layer, which
// paces the rows, runs ahead of a tile's last stage, where the marks are read.
constexpr int kMlpMarks = 8;

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
    int wide;                        // the first layer in units of 128 columns (else blocks of 64)
    float inv_d;
    uint32_t idesc_block, idesc_unit, idesc2;
};

// Shared-memory plan (byte offsets from the 1024-aligned dynamic base).
struct MlpPlan {
    uint32_t a, wm, w2, hid, term, anc, onehot, ident, bias, gamma, beta, stats, u, poison, prow, arow, total;
};

// Anchor segments of one block: the anchors of both of the pair's tiles, this CTA's half of the columns.
__host__ __device__ inline uint32_t mlp_anchor_bytes(int k_shift) { return 2u * (kBM >> k_shift) * (kMlpHC / 2) * 2u; }

__host__ __device__ inline MlpPlan mlp_plan(int rdim, int cols, int outs, int wide, int term_stages, int wm_stages,
                                            int w2_stages, int k_shift) {
    MlpPlan p;
    uint32_t off = 0;
    p.a = off;      off += static_cast<uint32_t>(rdim / kBK) * kMlpBlock;
    p.wm = off;     off += static_cast<uint32_t>(wm_stages * (rdim / kBK)) * ((wide ? 2 : 1) * kMlpHC / kG) * 128u;
    p.w2 = off;     off += static_cast<uint32_t>(w2_stages) * ((cols > 256 ? cols / 2 : cols) / kG) * 128u;
    p.hid = off;    off += static_cast<uint32_t>(kMlpHidden * outs) * kMlpBlock;
    p.term = off;   off += static_cast<uint32_t>(term_stages) * kMlpBlock;
    p.anc = off;    off += static_cast<uint32_t>(term_stages) * mlp_anchor_bytes(k_shift);
    off = (off + 1023u) & ~1023u;
    p.onehot = off; off += kBM * (2u * (kBM >> k_shift)) * 2u;
    off = (off + 1023u) & ~1023u;
    p.ident = off;  off += (kMlpHC / 2) * 128u;
    p.bias = off;   off += static_cast<uint32_t>(cols) * 4u;
    p.gamma = off;  off += static_cast<uint32_t>(cols) * 4u;
    p.beta = off;   off += static_cast<uint32_t>(cols) * 4u;
    p.stats = off;  off += static_cast<uint32_t>(4 * outs) * kBM * 8u;
    p.u = off;      off += 3u * kBM * 4u;
    p.poison = off; off += static_cast<uint32_t>(kMlpMarks) * (kBM >> k_shift) * 4u;
    p.prow = off;   off += 2u * kBM * 4u;
    p.arow = off;   off += 4u * (kBM >> k_shift) * 4u;
    p.total = off;
    return p;
}

struct MlpBars {
    unsigned long long a_full, a_empty, d2_full, d2_empty, stats_full, rows_full[2], u_full[3], u_empty[3];
    unsigned long long d1_full[2], d1_empty[2], wm_full[2], wm_empty[2];
    unsigned long long w2_full[kMlpMaxStages], w2_empty[kMlpMaxStages];
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
__device__ __forceinline__ void mlp_arrive_leader(uint32_t bar, uint32_t leader) { mlp_arrive_remote(mlp_peer(bar, leader)); }
// Completes `bar` once this thread's cp.async copies so far have landed (one of its expected arrivals).
__device__ __forceinline__ void mlp_cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
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
// Marks the anchors r (bit 0 of `which`) and r + 32 (bit 1) of a CTA pair's two tiles in the CTA of their tile: NaN at
// `marks` + anchor, visible there before anything that this thread announces afterwards.
__device__ __noinline__ void mlp_mark(uint32_t marks, uint32_t leader, int anchors, int r, uint32_t which) {
    for (int i = 0; i < 2; ++i, r += 32)
        if (which >> i & 1) {
            const int of = r >= anchors ? 1 : 0;
            asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(mlp_peer(marks + 4u * (r - of * anchors), leader + of)), "r"(0x7fc00000) : "memory");
        }
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
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
template <int kRegs>
__device__ __forceinline__ void mlp_more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs)); }
template <int kRegs>
__device__ __forceinline__ void mlp_fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs)); }
__device__ __forceinline__ void mlp_bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Whether one of eight 16-bit values is an infinity or NaN (an exponent of all ones).
template <int kDt>
__device__ __forceinline__ bool mlp_not_finite(const uint4& v) {
    constexpr uint32_t kExp = kDt == RLM_BF16 ? 0x7f807f80u : 0x7c007c00u, kUnit = kDt == RLM_BF16 ? 0x00800080u : 0x04000400u;
    const uint32_t carry = ((v.x & kExp) + kUnit) | ((v.y & kExp) + kUnit) | ((v.z & kExp) + kUnit) | ((v.w & kExp) + kUnit);
    return (carry & 0x80008000u) != 0;
}

// ---- tcgen05 on CTA pairs
//
// The issuing warps run their loops and waits with all lanes and predicate each tcgen05 instruction on one
// elected lane.  Inside an `if (lane == 0)` the compiler has to move every descriptor from vector to
// uniform registers one instruction at a time: 140 cycles per MMA, longer than most of them take.

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

// Shared-memory matrix descriptor with explicit leading / stride byte offsets and layout type.
__device__ __forceinline__ uint64_t mlp_desc(uint32_t addr, uint32_t leading, uint32_t stride, uint32_t layout) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | static_cast<uint64_t>(leading >> 4) << 16 |
           static_cast<uint64_t>(stride >> 4) << 32 | static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(layout) << 61;
}

__device__ __forceinline__ void mlp_umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                         bool issue) {
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
__device__ __forceinline__ void mlp_commit(uint32_t bar, uint32_t mask, bool issue) {
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        "setp.ne.b32 q, %2, 0;\n"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
        "}\n"
        ::"r"(bar), "h"(static_cast<uint16_t>(mask)), "r"(static_cast<uint32_t>(issue)) : "memory");
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

// The second layer's values are rounded to 16 bits before the LayerNorm, as where they pass through memory.
template <int kDt>
__device__ __forceinline__ float2 mlp_round(float2 x) {
    const uint32_t w = pack2(x.x, x.y, kDt);
    if (kDt == RLM_BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// Sixteen columns of the second layer's rows: accumulator + bias, rounded.
template <int kDt>
__device__ __forceinline__ void mlp_raw(const uint32_t (&v)[16], const float* bias, float2 (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 b = *reinterpret_cast<const float4*>(bias + 4 * i);
        x[2 * i] = mlp_round<kDt>(__fadd2_rn(make_float2(b.x, b.y), make_float2(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]))));
        x[2 * i + 1] = mlp_round<kDt>(__fadd2_rn(make_float2(b.z, b.w), make_float2(__uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]))));
    }
}

// This warp's columns of a finished tile: the group's weighted sum of its rows, residual and store.
// `ur` = weight * rstd of this lane's row (0: the row contributes nothing, whatever it holds), `u_sum` and `urm_sum` =
// sums over the group of the weight and of ur * mean:
//   sum u LayerNorm(x) = gamma (sum ur x - urm_sum) + beta u_sum.
// The next chunk's residual and tensor-memory columns are requested before a chunk is summed.
template <int kLG, int kDt>
__device__ __forceinline__ void mlp_store_rows(uint32_t tmem, int cols, int lane, bool live, float ur, float u_sum, float urm_sum,
                                               const float* bias, const float* gamma, const float* beta,
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
    uint32_t v[16];
    tmem_ld16(tmem, v);
#pragma unroll 1
    for (int c = 0; c < cols; c += 16) {
        float res[kCols];
#pragma unroll
        for (int k = 0; k < kCols; ++k) res[k] = next[k];
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float2 x[8];
        mlp_raw<kDt>(v, bias + c, x);
        float y[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 p = __fmul2_rn(x[i], make_float2(ur, ur));
            y[2 * i] = ur == 0.0f ? 0.0f : p.x;
            y[2 * i + 1] = ur == 0.0f ? 0.0f : p.y;
        }
        if (c + 16 < cols) {
            tmem_ld16(tmem + static_cast<uint32_t>(c + 16), v);
            fetch(c + 16);
        } else {                                         // the accumulator may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (drained) mlp_arrive_remote(drained_bar);
        }
        mlp_group_sum<kLG>(y, lane);
        if (!store) continue;
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
            const int col = c + c0 + k;
            res[k] += fmaf(gamma[col], y[k] - urm_sum, beta[col] * u_sum);
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

template <int kDt>
__global__ void __launch_bounds__(kMlpThreads, 1) relation_mlp_rows_kernel(
    const __grid_constant__ CUtensorMap map_wm, const __grid_constant__ CUtensorMap map_w2,
    const MlpArgs a, const int outs) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) MlpBars bars;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed_s;
    volatile int* failed = &failed_s;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // warp-uniform
    const int C = outs, R = a.rdim, H = a.hdim, NC = a.cols, wide = a.wide;
    const uint32_t rank = mlp_rank();
    const int o = static_cast<int>(rank) / kG, g = static_cast<int>(rank) % kG;      // output part, row group
    const uint32_t leader = static_cast<uint32_t>(o * kG);                           // issues the pair's MMAs
    const uint32_t pair_mask = ((1u << kG) - 1u) << leader;
    const int kblocks = R / kBK, U = H / (2 * kMlpHC * C);                           // units of 128 hidden columns per CTA
    const int cluster = static_cast<int>(blockIdx.x) / (C * kG), n_clusters = static_cast<int>(gridDim.x) / (C * kG);
    const int n_super = (a.n_tiles + kG - 1) / kG;
    const int anchors = kBM >> a.k_shift, sel_k = kG * anchors;                      // anchors of a tile, of the pair

    unsigned char* base = smem_align1024(smem_raw);
    const MlpPlan plan = mlp_plan(R, NC, C, wide, a.term_stages, a.wm_stages, a.w2_stages, a.k_shift);
    const uint32_t s_a = smem_u32(base + plan.a), s_wm = smem_u32(base + plan.wm), s_w2 = smem_u32(base + plan.w2);
    const uint32_t s_hid = smem_u32(base + plan.hid), s_term = smem_u32(base + plan.term), s_anc = smem_u32(base + plan.anc);
    const uint32_t anc_stage = mlp_anchor_bytes(a.k_shift);
    const int wm_rows = (wide ? 2 : 1) * kMlpHC / kG;                                // weight rows of a stage in this CTA
    const uint32_t wm_kblock = static_cast<uint32_t>(wm_rows) * 128u, wm_stage = static_cast<uint32_t>(kblocks) * wm_kblock;
    const int n_inst = NC > 256 ? 2 : 1, NI = NC / n_inst;
    const uint32_t w2_stage = static_cast<uint32_t>(NI / kG) * 128u;                 // one instruction's weight rows
    float* bias_s = reinterpret_cast<float*>(base + plan.bias);
    float* gamma_s = reinterpret_cast<float*>(base + plan.gamma);
    float* beta_s = reinterpret_cast<float*>(base + plan.beta);
    float2* stats_s = reinterpret_cast<float2*>(base + plan.stats);
    float* u_s = reinterpret_cast<float*>(base + plan.u);
    int* prow_s = reinterpret_cast<int*>(base + plan.prow);
    int* arow_s = reinterpret_cast<int*>(base + plan.arow);
    float* poison_s = reinterpret_cast<float*>(base + plan.poison);      // [kMlpMarks tiles in turn][anchor]: 0, or NaN for one that is not finite

    if (tid == 0) {
        failed_s = 0;
        const auto init = [](unsigned long long* b, int count) { mbar_init(smem_u32(b), static_cast<uint32_t>(count)); };
        // what the leader waits for from both CTAs: its own arrival and the one that the other CTA forwards
        const int both = g == 0 ? 2 : 1;
        init(&bars.a_full, kMlpOperandWarps * kG);
        init(&bars.a_empty, 1);
        init(&bars.d2_full, 1);
        init(&bars.d2_empty, kMlpEpiWarps * kG);
        init(&bars.stats_full, C == 1 ? kMlpEpiWarps : 1);
        for (int i = 0; i < 3; ++i) {
            init(&bars.u_full[i], kBM / 32);
            init(&bars.u_empty[i], kMlpEpiWarps);
        }
        for (int i = 0; i < 2; ++i) {
            init(&bars.rows_full[i], kBM / 32);
            init(&bars.d1_full[i], 1);
            init(&bars.d1_empty[i], (wide ? kMlpEpiWarps : kMlpEpiWarps / 2) * kG);
            init(&bars.wm_full[i], both);
            init(&bars.wm_empty[i], 1);
        }
        for (int i = 0; i < kMlpMaxStages; ++i) {
            init(&bars.w2_full[i], both);
            init(&bars.w2_empty[i], 1);
        }
        for (int i = 0; i < kMlpHidden; ++i) {
            for (int b = 0; b < 2; ++b) init(&bars.hid_full[i][b], C == 1 ? kMlpEpiWarps / 2 : 4);
            init(&bars.hid_empty[i], C);
        }
        for (int i = 0; i < kMlpMaxTerms; ++i) {
            init(&bars.term_full[i], (32 + 1) * kMlpGatherWarps + both - 1);
            init(&bars.term_empty[i], 1);
        }
        fence_barrier_init();
    }
    if (warp == kMlpEpiWarps + 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < NC; i += kMlpThreads) {       // parameters of this CTA's output columns
        bias_s[i] = a.second_bias[o * NC + i];
        gamma_s[i] = a.norm_w[o * NC + i];
        beta_s[i] = a.norm_b[o * NC + i];
    }
    for (int i = tid; i < kMlpMarks * anchors; i += kMlpThreads) poison_s[i] = 0.0f;
    const uint16_t one = kDt == RLM_BF16 ? 0x3f80 : 0x3c00;
    for (int i = tid; i < kBM * sel_k / 8; i += kMlpThreads) {          // one-hot rows: K-chunk major core matrices, no swizzle
        const int c = i / kBM, r = i - c * kBM;
        const int hot = g * anchors + (r >> a.k_shift) - 8 * c;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = hot >> 1 == e && hot >= 0 ? static_cast<uint32_t>(one) << (16 * (hot & 1)) : 0u;
        *reinterpret_cast<uint4*>(base + plan.onehot + c * (kBM * 16) + r * 16) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    for (int i = tid; i < (kMlpHC / kG) * 8; i += kMlpThreads) {        // this CTA's half of the 64 x 64 identity
        const int r = i >> 3, c = i & 7, hot = g * (kMlpHC / kG) + r - 8 * c;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = hot >> 1 == e && hot >= 0 ? static_cast<uint32_t>(one) << (16 * (hot & 1)) : 0u;
        *reinterpret_cast<uint4*>(base + plan.ident + swizzled(r, c, kMlpBlock)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    fence_proxy_async();
    griddep_sync();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    mlp_cluster_sync();                                  // every CTA's barriers are initialised
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d2 = __shfl_sync(0xffffffffu, tmem_slot, 0), tmem_d1 = tmem_d2 + static_cast<uint32_t>(NC);
    // hidden column of block n (64 columns, counted within a tile) of part b
    const auto column = [&](int n, int b) { return ((n >> 1) * C + b) * (2 * kMlpHC) + (n & 1) * kMlpHC; };

    if (warp < kMlpEpiWarps) {
        mlp_more_registers<kMlpEpiRegs>();
        // ------------------------------------------------------------ epilogue
        // Two groups of eight warps take the two blocks of a unit; thread = pair row x 32 of a block's 64 columns.
        const int row = 32 * (warp & 3) + lane, turn = warp >> 3, half = (warp >> 2) & 1;
        const uint32_t lane_base = static_cast<uint32_t>(32 * (warp & 3)) << 16;
        unsigned char* block = base + plan.hid + static_cast<uint32_t>(turn * C + o) * kMlpBlock;
        // this thread's chunk c of the block lies at cell ^ (c << 4): 128-byte rows, chunks swizzled by the row
        const uint32_t cell = smem_u32(block) + static_cast<uint32_t>((row >> 3) * 1024 + (row & 7) * 128 + (((4 * half) ^ (row & 7)) << 4));
        const uint32_t full = smem_u32(&bars.hid_full[turn][o]), part = smem_u32(block) + static_cast<uint32_t>(warp & 3) * 4096u;
        const int q = warp >> 2, quarter = NC / 4;                   // output columns of this warp in the last stage
        const int group = 1 << a.group_shift;
        const uint32_t d2_drained = mlp_peer(smem_u32(&bars.d2_empty), leader);
        const uint32_t d1_at = tmem_d1 + lane_base + static_cast<uint32_t>(turn * kMlpHC + 32 * half);
        int unit = 0, tix = 0, tix3 = 0, u_phase = 0;
        bool ok = true;
        const auto hidden_block = [&]() {
            const int buffer = wide ? unit & 1 : turn, phase = wide ? (unit >> 1) & 1 : unit & 1;
            ok = ok && mlp_wait(smem_u32(&bars.d1_full[buffer]), phase, failed);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t from = d1_at + (wide ? static_cast<uint32_t>(buffer * 2 * kMlpHC) : 0u);
            uint4 w[4];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[16];
                tmem_ld16(from + 16 * hh, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (hh == 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (ok && lane == 0) mlp_arrive_leader(smem_u32(&bars.d1_empty[buffer]), leader);
                }
                uint32_t y[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 h = gelu_pair(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
                    y[i] = pack2(h.x, h.y, kDt);
                }
                w[2 * hh] = make_uint4(y[0], y[1], y[2], y[3]);
                w[2 * hh + 1] = make_uint4(y[4], y[5], y[6], y[7]);
            }
            // the block's previous content has been consumed, here and where it was copied to
            ok = ok && mlp_wait(smem_u32(&bars.hid_empty[turn]), (unit & 1) ^ 1, failed);
#pragma unroll
            for (int c = 0; c < 4; ++c)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                             ::"r"(cell ^ static_cast<uint32_t>(c << 4)), "r"(w[c].x), "r"(w[c].y), "r"(w[c].z), "r"(w[c].w) : "memory");
            fence_proxy_async();                                  // the block -> tensor core, bulk copy
            if (C == 1) {
                __syncwarp();
                if (ok && lane == 0) mlp_arrive(full);
            } else {
                // both warps of these 32 rows have written their columns: 4 KB that are contiguous in the block
                mlp_bar_sync(1 + 4 * turn + (warp & 3), 64);
                if (ok && half == 0 && lane == 0) {
                    mlp_arrive(full);
                    const uint32_t to = static_cast<uint32_t>((1 - o) * kG + g), bar = mlp_peer(full, to);
                    mlp_expect_remote(bar, 4096u);
                    mlp_copy_cluster(mlp_peer(part, to), part, 4096u, bar);
                }
            }
            ++unit;
        };
        // The next tile's first unit comes before a tile's last stage: its arithmetic falls into the second layer's
        // tail, and the second layer finds it ready.
        if (cluster < n_super) hidden_block();
        for (int super = cluster; super < n_super; super += n_clusters, ++tix) {
            for (int j = 1; j < U; ++j) hidden_block();
            if (super + n_clusters < n_super) hidden_block();
            // ---- the tile's second layer is complete: LayerNorm over d, weighted sum over the group
            const int tile = super * kG + g;
            const uint32_t tmem_row = tmem_d2 + lane_base + static_cast<uint32_t>(q * quarter);
            const float* bias = bias_s + q * quarter;
            ok = ok && mlp_wait(smem_u32(&bars.d2_full), tix & 1, failed);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (C > 1 && ok && tid == 0) mbar_expect_tx(smem_u32(&bars.stats_full), static_cast<uint32_t>(4 * C * kBM * 8));
            // statistics of this thread's columns about the mean of the first sixteen: one pass over the accumulator
            float shift = 0.0f, s1 = 0.0f, s2 = 0.0f;
            {
                uint32_t v[16];
                tmem_ld16(tmem_row, v);
#pragma unroll 1
                for (int c = 0; c < quarter; c += 16) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float2 x[8];
                    mlp_raw<kDt>(v, bias + c, x);
                    if (c + 16 < quarter) tmem_ld16(tmem_row + static_cast<uint32_t>(c + 16), v);
                    if (c == 0) {
                        float2 sum = x[0];
#pragma unroll
                        for (int i = 1; i < 8; ++i) sum = __fadd2_rn(sum, x[i]);
                        shift = (sum.x + sum.y) * 0.0625f;
                    }
                    float2 t1 = make_float2(0.0f, 0.0f), t2 = t1;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 y = __fadd2_rn(x[i], make_float2(-shift, -shift));
                        t1 = __fadd2_rn(t1, y);
                        t2 = __ffma2_rn(y, y, t2);
                    }
                    s1 += t1.x + t1.y;
                    s2 += t2.x + t2.y;
                }
            }
            const float inv_quarter = 1.0f / static_cast<float>(quarter);
            // (a row whose anchor is not finite becomes NaN here, and through the statistics in every output part)
            const float mean_q = fmaf(s1, inv_quarter, shift) + *static_cast<volatile float*>(poison_s + (tix & (kMlpMarks - 1)) * anchors + (row >> a.k_shift));
            const float m2 = fmaf(-s1 * inv_quarter, s1, s2);
            // every CTA of the tile receives (mean, sum of squares) of all quarters
            float2* mine = stats_s + (o * 4 + q) * kBM + row;
            if (C == 1) {
                *mine = make_float2(mean_q, m2);
                __syncwarp();
                if (ok && lane == 0) mlp_arrive(smem_u32(&bars.stats_full));
                ok = ok && mlp_wait(smem_u32(&bars.stats_full), tix & 1, failed);
            } else {
#pragma unroll
                for (int other = 0; other < 2; ++other) {
                    const uint32_t to = static_cast<uint32_t>(other * kG + g);
                    if (ok) mlp_store_remote(mlp_peer(smem_u32(mine), to), mean_q, m2, mlp_peer(smem_u32(&bars.stats_full), to));
                }
                ok = ok && mlp_wait<true>(smem_u32(&bars.stats_full), tix & 1, failed);
            }
            float2 st[8];
            float mean = 0.0f, total = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                st[i] = i < 4 * C ? stats_s[i * kBM + row] : make_float2(0.0f, 0.0f);
                mean += st[i].x;
            }
            mean *= C == 1 ? 0.25f : 0.125f;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i < 4 * C) total += fmaf(static_cast<float>(quarter) * (st[i].x - mean), st[i].x - mean, st[i].y);
            const float rstd = rsqrtf(fmaf(total, a.inv_d, a.eps));
            ok = ok && mlp_wait(smem_u32(&bars.u_full[tix3]), u_phase, failed);
            const float u = u_s[tix3 * kBM + row];
            __syncwarp();
            if (ok && lane == 0) mlp_arrive(smem_u32(&bars.u_empty[tix3]));
            if (++tix3 == 3) { tix3 = 0; u_phase ^= 1; }
            const float ur = u == 0.0f ? 0.0f : u * rstd;
            float u_sum = u, urm_sum = u == 0.0f ? 0.0f : ur * mean;
            for (int s = 1; s < group; s <<= 1) {
                u_sum += __shfl_xor_sync(0xffffffffu, u_sum, s);
                urm_sum += __shfl_xor_sync(0xffffffffu, urm_sum, s);
            }
            const int pair = tile * kBM + row;
            const bool live = ok && pair < a.n_pairs;
            const size_t at = (live ? static_cast<size_t>(pair >> a.group_shift) : 0) * a.d + static_cast<size_t>(o * NC + q * quarter);
            const float* res = a.residual ? a.residual + at : nullptr;
            const float *gm = gamma_s + q * quarter, *bt = beta_s + q * quarter;
            float* out = a.out + at;
            const bool drained = ok && lane == 0;
#define MLP_STORE(kLG) mlp_store_rows<kLG, kDt>(tmem_row, quarter, lane, live, ur, u_sum, urm_sum, bias, gm, bt, res, out, d2_drained, drained)
            switch (a.group_shift) {
                case 2: MLP_STORE(2); break;
                case 3: MLP_STORE(3); break;
                case 4: MLP_STORE(4); break;
                default: MLP_STORE(5); break;
            }
#undef MLP_STORE
        }
    } else if (warp == kMlpEpiWarps) {
        mlp_fewer_registers<kMlpIssueRegs>();
        // ------------------------------------------------------------ W_2 tiles
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w2) : "memory");
            int ws = 0, wphase = 0;
            bool ok = true;
            for (int super = cluster; ok && super < n_super; super += n_clusters)
                for (int n = 0; ok && n < 2 * U; ++n)
                    for (int p = 0; p < C; ++p)
                        for (int i = 0; i < n_inst; ++i) {
                            const uint32_t bar = smem_u32(&bars.w2_full[ws]);
                            ok = ok && mlp_wait(smem_u32(&bars.w2_empty[ws]), wphase ^ 1, failed);
                            if (!ok) break;
                            mbar_expect_tx(bar, w2_stage);
                            tma_load_2d(s_w2 + ws * w2_stage, &map_w2, column(n, p == 0 ? o : 1 - o),
                                        o * NC + i * NI + g * (NI / kG), bar);
                            if (++ws == a.w2_stages) { ws = 0; wphase ^= 1; }
                        }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 1) {
        mlp_fewer_registers<kMlpIssueRegs>();
        // ------------------------------------------------------------ W_m tiles: a unit's or a block's rows
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_wm) : "memory");
            int ms = 0, mphase = 0;
            bool ok = true;
            for (int super = cluster; ok && super < n_super; super += n_clusters)
                for (int n = 0; n < 2 * U; n += 1 + wide) {
                    const uint32_t bar = smem_u32(&bars.wm_full[ms]);
                    ok = ok && mlp_wait(smem_u32(&bars.wm_empty[ms]), mphase ^ 1, failed);
                    if (!ok) break;
                    mbar_expect_tx(bar, wm_stage);
                    for (int kb = 0; kb < kblocks; ++kb)
                        tma_load_2d(s_wm + ms * wm_stage + kb * wm_kblock, &map_wm, kb * kBK, column(n, o) + g * wm_rows, bar);
                    if (++ms == a.wm_stages) { ms = 0; mphase ^= 1; }
                }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 2) {
        mlp_fewer_registers<kMlpIssueRegs>();
        // ------------------------------------------------------------ first layer: D1 = segments + products x W_m rows
        const bool elected = mlp_elect(), issue = g == 0;
        const uint64_t a_desc = smem_desc_sw128(s_a), w_desc = smem_desc_sw128(s_wm);
        const uint64_t t_desc = smem_desc_sw128(s_term), i_desc = smem_desc_sw128(smem_u32(base + plan.ident));
        // one-hot rows: 128-byte core matrices, K chunks 16 * 128 bytes apart, 8-row groups 128 bytes apart, no swizzle
        const uint64_t s_desc = mlp_desc(smem_u32(base + plan.onehot), kBM * 16, 128, 0);
        // anchor segments [anchor][32 columns]: N-major, 64-byte swizzle, 8-anchor groups 512 bytes apart
        const uint64_t n_desc = mlp_desc(s_anc, 16, 512, 4);
        const int sel_steps = sel_k / 16;
        int ms = 0, mphase = 0, ts = 0, tphase = 0, unit = 0, tix = 0;
        bool ok = true;
        const auto products = [&](uint32_t d_at, uint32_t idesc, int buffer) {
            ok = ok && mlp_wait(smem_u32(&bars.wm_full[ms]), mphase, failed);
            if (issue) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const bool go = elected && ok;
                const uint64_t wd = w_desc + (static_cast<uint32_t>(ms) * wm_stage >> 4);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk) mlp_umma(d_at, a_desc + 2 * kk, wd + 2 * kk, idesc, 1u, go);
                if (kblocks > 1)
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)
                        mlp_umma(d_at, a_desc + (kMlpBlock >> 4) + 2 * kk, wd + (wm_kblock >> 4) + 2 * kk, idesc, 1u, go);
                mlp_commit(smem_u32(&bars.d1_full[buffer]), pair_mask, go);
                mlp_commit(smem_u32(&bars.wm_empty[ms]), pair_mask, go);
            } else if (ok && elected) {
                mlp_arrive_leader(smem_u32(&bars.wm_full[ms]), leader);
            }
            if (++ms == a.wm_stages) { ms = 0; mphase ^= 1; }
        };
        for (int super = cluster; ok && super < n_super; super += n_clusters, ++tix) {
            for (int j = 0; ok && j < U; ++j, ++unit) {
                const uint32_t unit_at = tmem_d1 + (wide ? static_cast<uint32_t>((unit & 1) * 2 * kMlpHC) : 0u);
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const uint32_t d_at = unit_at + static_cast<uint32_t>(s * kMlpHC);
                    if (issue && (s == 0 || !wide))
                        ok = ok && mlp_wait(smem_u32(&bars.d1_empty[wide ? unit & 1 : s]), (wide ? (unit >> 1) & 1 : unit & 1) ^ 1, failed);
                    ok = ok && mlp_wait(smem_u32(&bars.term_full[ts]), tphase, failed);
                    fence_proxy_async();              // the segments came by ordinary (cp.async) writes
                    if (issue) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const bool go = elected && ok;
                        const uint64_t td = t_desc + (static_cast<uint32_t>(ts) * kMlpBlock >> 4);
                        const uint64_t nd = n_desc + (static_cast<uint32_t>(ts) * anc_stage >> 4);
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; ++kk)
                            mlp_umma(d_at, td + 2 * kk, i_desc + 2 * kk, a.idesc_block, kk > 0 ? 1u : 0u, go);
                        for (int kk = 0; kk < sel_steps; ++kk)
                            mlp_umma(d_at, s_desc + kk * (2 * kBM * 16 >> 4), nd + kk * (1024 >> 4), a.idesc_block | (1u << 16), 1u, go);
                        mlp_commit(smem_u32(&bars.term_empty[ts]), pair_mask, go);
                    } else if (ok && elected) {
                        mlp_arrive_leader(smem_u32(&bars.term_full[ts]), leader);
                    }
                    if (++ts == a.term_stages) { ts = 0; tphase ^= 1; }
                    if (s == 0 && j == 0 && issue) ok = ok && mlp_wait(smem_u32(&bars.a_full), tix & 1, failed);
                    if (!wide) products(d_at, a.idesc_block, s);
                }
                if (wide) products(unit_at, a.idesc_unit, unit & 1);
                if (issue && j + 1 == U) mlp_commit(smem_u32(&bars.a_empty), pair_mask, elected && ok);
            }
        }
        __syncwarp();
    } else if (warp == kMlpEpiWarps + 3) {
        mlp_fewer_registers<kMlpIssueRegs>();
        // ------------------------------------------------------------ second layer: D2 += hidden blocks x W_2 columns
        const bool elected = mlp_elect(), issue = g == 0;
        const uint64_t h_desc = smem_desc_sw128(s_hid), w_desc = smem_desc_sw128(s_w2);
        int ws = 0, wphase = 0, unit = 0, tix = 0;
        bool ok = true;
        for (int super = cluster; ok && super < n_super; super += n_clusters, ++tix) {
            if (issue) ok = ok && mlp_wait(smem_u32(&bars.d2_empty), (tix & 1) ^ 1, failed);
            for (int n = 0; ok && n < 2 * U; ++n) {
                const int d = n & 1, phase = (unit + (n >> 1)) & 1;
                for (int p = 0; p < C; ++p) {
                    const int b = p == 0 ? o : 1 - o;          // this CTA's own block first: the other one is still on its way
                    ok = ok && mlp_wait(smem_u32(&bars.hid_full[d][b]), phase, failed);
                    const uint64_t hd = h_desc + (static_cast<uint32_t>(d * C + b) * kMlpBlock >> 4);
                    for (int i = 0; i < n_inst; ++i) {
                        ok = ok && mlp_wait(smem_u32(&bars.w2_full[ws]), wphase, failed);
                        if (issue) {
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const bool go = elected && ok;
                            const uint64_t wd = w_desc + (static_cast<uint32_t>(ws) * w2_stage >> 4);
#pragma unroll
                            for (int kk = 0; kk < kBK / 16; ++kk)
                                mlp_umma(tmem_d2 + static_cast<uint32_t>(i * NI), hd + 2 * kk, wd + 2 * kk, a.idesc2,
                                         (n > 0 || p > 0 || kk > 0) ? 1u : 0u, go);
                            mlp_commit(smem_u32(&bars.w2_empty[ws]), pair_mask, go);
                            if (i + 1 == n_inst) mlp_commit(smem_u32(&bars.hid_empty[d]), ((1u << kG) - 1u) << (b * kG), go);
                        } else if (ok && elected) {
                            mlp_arrive_leader(smem_u32(&bars.w2_full[ws]), leader);      // this CTA's block and weight rows are there
                        }
                        if (++ws == a.w2_stages) { ws = 0; wphase ^= 1; }
                    }
                }
            }
            unit += U;
            if (issue) mlp_commit(smem_u32(&bars.d2_full), pair_mask, elected && ok);
        }
        __syncwarp();
    } else if (warp < kMlpEpiWarps + 4 + kMlpGatherWarps) {
        mlp_fewer_registers<kMlpIssueRegs>();
        // ------------------------------------------------------------ expanded-cache segments of every block
        // 64 columns of the tile's 128 partner rows (128-byte swizzle), this CTA's 32 of the 64 columns of the pair's
        // anchor rows (64-byte swizzle), a thread per 16-byte chunk.  The anchors' chunks are requested a block ahead
        // into registers, where they are looked at (see the top).  What that costs, and the other places measured for
        // it, as us a pass of 8 x 4096 rows of d 512: 1266 without looking, 1300 here; the operand warps over the
        // anchors' whole rows 1306 (another read of them); the issuing warp 1433 (in the way of every block's products).
        const int gt = tid - 32 * (kMlpEpiWarps + 4), c = gt & 7, ac = gt & 3;
        const size_t ex_row = static_cast<size_t>(H) * 4;
        const char* expanded = static_cast<const char*>(a.expanded_cache);
        const char* partners = expanded + static_cast<size_t>(H) * 2 + 16 * c;
        const uint32_t to = swizzled(gt >> 3, c, kMlpBlock);               // rows 16 apart: 2048 bytes apart
        const uint32_t anchor_to = static_cast<uint32_t>((gt >> 2) * 64 + ((ac ^ ((gt >> 3) & 3)) << 4));      // ... 32 apart alike
        int ts = 0, tphase = 0, tix = 0;
        bool ok = true;
        for (int super = cluster; super < n_super; super += n_clusters, ++tix) {
            ok = ok && mlp_wait(smem_u32(&bars.rows_full[tix & 1]), (tix >> 1) & 1, failed);
            int prow[8], arow[2];
#pragma unroll
            for (int i = 0; i < 8; ++i) prow[i] = prow_s[(tix & 1) * kBM + (gt >> 3) + 16 * i];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = (gt >> 2) + 8 * kMlpGatherWarps * i;
                arow[i] = r < sel_k ? arow_s[(tix & 1) * sel_k + r] : -1;
            }
            uint4 ahead[2];
            uint32_t bad = 0;                                     // this thread's anchors that are not finite
            const auto request_anchors = [&](int n) {
                const char* from = expanded + static_cast<size_t>(column(n, o)) * 2 + g * (kMlpHC / kG) * 2 + 16 * ac;
#pragma unroll
                for (int i = 0; i < 2; ++i) {      // beyond the last row: every row's product reads it (times zero)
                    ahead[i] = make_uint4(0, 0, 0, 0);
                    if (arow[i] >= 0) ahead[i] = *reinterpret_cast<const uint4*>(from + arow[i] * ex_row);
                }
            };
            if (ok) request_anchors(0);
            for (int n = 0; n < 2 * U; ++n) {
                const size_t h_bytes = static_cast<size_t>(column(n, o)) * 2;
                const uint32_t block = s_term + static_cast<uint32_t>(ts) * kMlpBlock + to;
                ok = ok && mlp_wait(smem_u32(&bars.term_empty[ts]), tphase ^ 1, failed);
                if (ok) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (prow[i] >= 0) cp_async16(block + 2048u * i, partners + prow[i] * ex_row + h_bytes);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int r = (gt >> 2) + 8 * kMlpGatherWarps * i;
                        if (r >= sel_k) break;
                        if (mlp_not_finite<kDt>(ahead[i])) {
                            ahead[i] = make_uint4(0, 0, 0, 0);
                            bad |= 1u << i;
                        }
                        *reinterpret_cast<uint4*>(base + plan.anc + static_cast<uint32_t>(ts) * anc_stage + anchor_to + 2048u * i) = ahead[i];
                    }
                    if (n + 1 < 2 * U) request_anchors(n + 1);
                    else if (bad) mlp_mark(smem_u32(poison_s + (tix & (kMlpMarks - 1)) * anchors), leader, anchors, gt >> 2, bad);
                    mlp_cp_async_arrive(smem_u32(&bars.term_full[ts]));
                }
                __syncwarp();                                 // the warp's stores -> its one arrival for them
                if (ok && lane == 0) mlp_arrive(smem_u32(&bars.term_full[ts]));
                if (++ts == a.term_stages) { ts = 0; tphase ^= 1; }
            }
        }
        cp_async_wait_all();
    } else {
        mlp_fewer_registers<kMlpOperandRegs>();
        // ------------------------------------------------------------ indices, weights and operand products
        const int gt = tid - 32 * (kMlpEpiWarps + 4 + kMlpGatherWarps), gw = gt >> 5;
        const int K = 1 << a.k_shift, chunks = R / 8, rows_per_warp = 32 / chunks;
        const size_t op_row = static_cast<size_t>(R) * 2;
        const char* operand = static_cast<const char*>(a.operand_cache);
        const int cc = lane % chunks, r_first = gw * rows_per_warp + lane / chunks, r_step = kMlpOperandWarps * rows_per_warp;
        int tix = 0, u_at = 0, u_phase = 0, made = 0;
        bool ok = true;
        // Tile `super`'s cache rows (its partners; the anchors of both of the pair's tiles) into buffer `b`.
        const auto rows = [&](int super, int b) {
            if (gt >= kBM) return;                           // the first four warps, a pair each
            const int pair = (super * kG + g) * kBM + gt;
            int prow = -1;
            if (pair < a.n_pairs)
                prow = (pair >> a.k_shift) / a.slots / a.rows_per_seq * a.max_t + min(max(a.partner_index[pair], 0), a.max_t - 1);
            prow_s[b * kBM + gt] = prow;
            if (gt < sel_k) {
                const int srow = super * sel_k + gt;
                int arow = -1;
                if (srow < a.n_pairs >> a.k_shift)
                    arow = srow / a.slots / a.rows_per_seq * a.max_t + min(max(a.anchor_index[srow], 0), a.max_t - 1);
                arow_s[b * sel_k + gt] = arow;
            }
            // The next tile's marks: the slot was the tile's seven before this one, which the epilogue has read (`weights` of
            // two tiles ago waited for the tile five before); nothing of the next tile is gathered before this one is announced.
            ++made;
            if (gt < anchors) poison_s[(made & (kMlpMarks - 1)) * anchors + gt] = 0.0f;
            __syncwarp();
            if (ok && lane == 0) mlp_arrive(smem_u32(&bars.rows_full[b]));
        };
        // This thread's pair's weight into u: first wanted in the tile's last stage, so behind everything that the tile's
        // products wait for (a pass of 512 rows of d 256, where a tile is all there is: 57.7 -> 55.6 us).
        const auto weights = [&](int super) {
            if (gt >= kBM) return;
            const int pair = (super * kG + g) * kBM + gt;
            float u = 0.0f;
            if (pair < a.n_pairs) {
                const int srow = pair >> a.k_shift, k = pair & (K - 1);
                const int query = srow / a.slots, slot = srow - query * a.slots;
                int k_limit = K;
                if (a.limited) k_limit = min(max(32 - __clz(query - query / a.rows_per_seq * a.rows_per_seq + 1), 1), K);      // ceil(log2(t + 2))
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
            // The weights are read in a tile's last stage, the first layer runs ahead of it: with two or three units a
            // tile the slot may still be waiting to be read.
            ok = ok && mlp_wait(smem_u32(&bars.u_empty[u_at]), u_phase ^ 1, failed);
            u_s[u_at * kBM + gt] = u;
            __syncwarp();
            if (ok && lane == 0) mlp_arrive(smem_u32(&bars.u_full[u_at]));
            if (++u_at == 3) { u_at = 0; u_phase ^= 1; }
        };
        if (cluster < n_super) rows(cluster, 0);
        for (int super = cluster; super < n_super; super += n_clusters, ++tix) {
            const int* prow_t = prow_s + (tix & 1) * kBM;
            const int* arow_t = arow_s + (tix & 1) * sel_k + g * anchors;
            mlp_bar_sync(9, 32 * kMlpOperandWarps);          // this tile's rows are written, the other buffer is no longer read
            // a lane per 16-byte chunk; the products wait in registers until the A tile is free
            uint4 product[8];
#pragma unroll
            for (int i0 = 0; i0 < 8; i0 += 2) {
                uint4 pv[2], av[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = r_first + (i0 + i) * r_step, prow = r < kBM ? prow_t[r] : -1;
                    pv[i] = av[i] = make_uint4(0, 0, 0, 0);
                    if (prow >= 0) {
                        pv[i] = *reinterpret_cast<const uint4*>(operand + prow * op_row + 16 * cc);
                        av[i] = *reinterpret_cast<const uint4*>(operand + arow_t[r >> a.k_shift] * op_row + 16 * cc);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float fp[8], fa[8];
                    unpack8(pv[i], kDt, fp);
                    unpack8(av[i], kDt, fa);
                    product[i0 + i] = make_uint4(pack2(fp[0] * fa[0], fp[1] * fa[1], kDt), pack2(fp[2] * fa[2], fp[3] * fa[3], kDt),
                                                 pack2(fp[4] * fa[4], fp[5] * fa[5], kDt), pack2(fp[6] * fa[6], fp[7] * fa[7], kDt));
                }
            }
            ok = ok && mlp_wait(smem_u32(&bars.a_empty), (tix & 1) ^ 1, failed);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = r_first + i * r_step;
                if (r < kBM) *reinterpret_cast<uint4*>(base + plan.a + swizzled(r, cc, kMlpBlock)) = product[i];
            }
            fence_proxy_async();
            __syncwarp();
            if (ok && lane == 0) mlp_arrive_leader(smem_u32(&bars.a_full), leader);
            if (super + n_clusters < n_super) rows(super + n_clusters, (tix & 1) ^ 1);
            weights(super);
        }
    }
    // ---- leave together: no CTA may go while another still reads or signals its shared memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    mlp_cluster_sync();
    if (tid == 0 && failed_s && a.status) atomicOr(a.status, RLM_DEV_TIMEOUT);
    if (warp == kMlpEpiWarps + 2)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_d2) : "memory");
}

// ------------------------------------------------------------------ host

struct MlpShape { int outs, cols, wide, term_stages, wm_stages, w2_stages; uint32_t smem; bool ok; };

bool power_of_two(int v) { return v > 0 && (v & (v - 1)) == 0; }

int log2_of(int v) {
    int s = 0;
    while ((1 << s) < v) ++s;
    return s;
}

// `spread`: two output parts also where one would do.
// Output columns per CTA (tensor memory: cols of the second layer + one or two units of the first) and the
// first of a list of pipeline depths that fits the shared memory.  At d = 512, K = 8, where two fit, two gathered
// blocks with three W_2 stages measured 745 us for 262 144 pairs, three with two 786 us.
MlpShape mlp_shape(int rdim, int hdim, int d, int k_shift, bool spread = false) {
    static constexpr int kDepths[][3] = {{4, 4, 2}, {3, 4, 2}, {3, 3, 2}, {3, 3, 1}, {2, 4, 1}, {2, 3, 1}, {2, 2, 1}};
    MlpShape s{};
    s.outs = d <= 384 && !spread ? 1 : 2;
    s.cols = d / s.outs;
    if (d % s.outs != 0 || s.cols % 64 != 0 || s.cols > 384 || hdim % (2 * kMlpHC * s.outs) != 0 || hdim < 4 * kMlpHC * s.outs) return s;
    s.wide = s.cols <= 256;
    for (const auto& depth : kDepths) {
        const MlpPlan p = mlp_plan(rdim, s.cols, s.outs, s.wide, depth[0], depth[2], depth[1], k_shift);
        if (p.total + 1024 > static_cast<uint32_t>(kSmemDynamicLimit)) continue;
        s.term_stages = depth[0];
        s.w2_stages = depth[1];
        s.wm_stages = depth[2];
        s.smem = p.total + 1024;
        s.ok = true;
        break;
    }
    return s;
}

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

template <int kDt>
int launch_mlp(const MlpArgs& a0, const MlpShape& s, const void* product_weight, const void* second_weight, void* stream) {
    MlpArgs a = a0;
    CUtensorMap map_wm, map_w2;
    const int n_inst = s.cols > 256 ? 2 : 1;
    if (!make_map(&map_wm, product_weight, a.hdim, a.rdim, a.rdim, (s.wide ? 2 : 1) * kMlpHC / kG, kDt) ||
        !make_map(&map_w2, second_weight, a.d, a.hdim, a.hdim, s.cols / n_inst / kG, kDt)) {
        set_error("relation_mlp_rows: tensor map encoding failed");
        return RLM_ERR_LAUNCH;
    }
    auto* kernel = relation_mlp_rows_kernel<kDt>;
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
    if (!power_of_two(k_out) || !power_of_two(slots) || k_out * slots > 32 || k_out < 4 || k_out > 16 || slots > 8) return 0;
    if (relation_dim != 64 && relation_dim != 128) return 0;
    if (d_model < 64 || hidden_dim < kMlpHC) return 0;
    return mlp_shape(relation_dim, hidden_dim, d_model, log2_of(k_out)).ok ? 1 : 0;
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
    MlpShape s = mlp_shape(relation_dim, hidden_dim, d_model, k_shift);
    // A launch that leaves more than half of the SMs idle divides its tiles' columns and hidden blocks over twice as many
    // CTAs, up to the 33 clusters of four that run at a time (us, one part -> two: 2048 pairs of d 256 31.5 -> 25.2, 4096
    // 31.7 -> 25.3, 8192 33.2 -> 27.4; beyond that a second wave would cost more).
    const int supers = (static_cast<int>((static_cast<int64_t>(n_rows) * slots * k_out + kBM - 1) / kBM) + kG - 1) / kG;
    if (s.outs == 1 && supers * 2 * kG <= sm_count() - 16) {
        const MlpShape spread = mlp_shape(relation_dim, hidden_dim, d_model, k_shift, true);
        if (spread.ok) s = spread;
    }
    const int n_inst = s.cols > 256 ? 2 : 1;
    const uint32_t fmt = dtype == RLM_BF16 ? 1u : 0u;
    const auto idesc = [&](int n) {
        return (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
               (static_cast<uint32_t>((kBM * kG) >> 4) << 24);
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
    a.wide = s.wide;
    a.inv_d = 1.0f / static_cast<float>(d_model);
    a.idesc_block = idesc(kMlpHC);
    a.idesc_unit = idesc(2 * kMlpHC);
    a.idesc2 = idesc(s.cols / n_inst);
    return dtype == RLM_BF16 ? launch_mlp<RLM_BF16>(a, s, product_weight, second_weight, stream)
                             : launch_mlp<RLM_F16>(a, s, product_weight, second_weight, stream);
}

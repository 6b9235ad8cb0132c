// Routed anchor/partner selection for sm_100a.
//
// One CTA per query row.  Everything a row needs is staged in shared memory by
// untiled bulk (TMA) copies that complete on mbarriers: both streams' block
// statistics and local key windows are requested at kernel entry; the chosen
// remote blocks are requested as soon as the block ranks are known, and the one
// partner-anchor cache row is read directly from global memory.  Key rows are
// scored from shared memory a lane per 64-wide row, block statistics with 8
// lanes per block (16-byte reads, bank-conflict free for 16-bit caches), in
// the canonical order documented in rlm_common.cuh, so the selected indices
// do not depend on the launch geometry.
//
// Semantics follow src/relation_lm/kernels/relation_select.py:50-308 and
// src/relation_lm/kernels/triton_select.py:23-252 of the reference project.

#include "relation_select_body.cuh"

namespace rlm {
namespace {

// kMinCtas = 3: the latency-oriented build (decode batches: one wave or less).  kMinCtas = 4:
// launches of many rows, where rows in flight per SM set the throughput.
template <int kMinCtas, int kDt, bool kDecode>
__global__ void __launch_bounds__(kThreads, kMinCtas) relation_select_kernel(const SelectArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    select_row<kDt, kDecode, false>(a, blockIdx.x, smem, smem_u32(smem + a.plan.bars));
}

// ---- routed multi-anchor selection: S anchor slots per query row, one launch
//
// Rules of the reference's dense multi-anchor layer (src/relation_lm/models/multi_relation_blocks.py)
// applied inside each slot's routed candidate set: slot s is active for a query at position t iff
// s <= t (:82-84); slots choose their anchors one after another and a position taken by an earlier
// slot is barred (:86-93); an inactive slot reports anchor 0 (:94); the partner selection of every
// slot bars the anchors of all active slots (:133-139); an inactive slot has no partners
// (:140-142); a partner slot is active iff its score is finite (:144-147).  Every slot has its own
// key caches, block statistics and router parameters (leading slot dimension).
constexpr int kMaxSlots = kMaxExclude;

struct MultiSelectArgs {
    SelectArgs base;               // slot 0's pointers; per-slot strides below (bytes)
    Plan plan_anchor, plan_partner;
    int slots;
    size_t keys_slot, pac_slot, stats_slot, gamma_slot, bias_slot;   // bytes between slots
    int32_t* out_anchor;           // [N, S]
    float* out_anchor_score;       // [N, S]
    uint8_t* out_anchor_active;    // [N, S]
    int32_t* out_partner;          // [N, S, K]
    float* out_partner_score;      // [N, S, K]
};

__device__ __forceinline__ const void* slot_ptr(const void* p, size_t bytes) {
    return static_cast<const char*>(p) + bytes;
}

template <int kDt>
__global__ void __launch_bounds__(kThreads, 3) relation_select_multi_kernel(const MultiSelectArgs m) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long call_bars[4 * 2 * kMaxSlots];
    __shared__ int taken_s[kMaxSlots];
    const int row = blockIdx.x, tid = threadIdx.x;
    const int S = m.slots, K = m.base.k_out;
    griddep_sync();
    const int b = m.base.row_batch[row], t = m.base.row_position[row];
    if (b < 0 || b >= m.base.n_seq || t < 0 || t >= m.base.max_t) {
        if (tid == 0 && m.base.status) atomicOr(m.base.status, RLM_DEV_POSITION);
        return;
    }
    if (tid < kMaxSlots) taken_s[tid] = -1;
    __syncthreads();
    const int esz = m.base.query_dtype == RLM_F32 ? 4 : 2;
    // anchors: slot after slot, each barring the positions taken before it
    for (int s = 0; s < S; ++s) {
        const bool slot_live = s <= t;
        int32_t* out_idx = m.out_anchor + static_cast<size_t>(row) * S + s;
        float* out_sc = m.out_anchor_score + static_cast<size_t>(row) * S + s;
        if (slot_live) {
            SelectArgs a = m.base;
            a.mode = kAnchorOnly;
            a.plan = m.plan_anchor;
            a.anchor_query = slot_ptr(m.base.anchor_query, static_cast<size_t>(s) * kD * esz);
            a.anchor_router_query = slot_ptr(m.base.anchor_router_query, static_cast<size_t>(s) * kD * esz);
            a.anchor_keys = slot_ptr(m.base.anchor_keys, s * m.keys_slot);
            a.anchor_mean = slot_ptr(m.base.anchor_mean, s * m.stats_slot);
            a.anchor_std = slot_ptr(m.base.anchor_std, s * m.stats_slot);
            a.anchor_gamma = slot_ptr(m.base.anchor_gamma, s * m.gamma_slot);
            a.anchor_bias = slot_ptr(m.base.anchor_bias, s * m.bias_slot);
            a.exclude_list = s > 0 ? taken_s - static_cast<ptrdiff_t>(row) * s : nullptr;   // [row * s + i] == taken_s[i]
            a.exclude_count = s;
            a.out_anchor = out_idx - row;                    // [row] lands on (row, s)
            a.out_anchor_score = out_sc - row;
            select_row<kDt, false, true>(a, row, smem, smem_u32(&call_bars[4 * s]));
        }
        __syncthreads();
        if (tid == 0) {                                      // the thread that stored the slot's result
            const bool live = slot_live && *out_sc > kNegInf;
            if (!live) { *out_idx = 0; *out_sc = kNegInf; }
            taken_s[s] = live ? *out_idx : -1;
            m.out_anchor_active[static_cast<size_t>(row) * S + s] = live ? 1 : 0;
        }
        __syncthreads();
    }
    // partners: every live slot bars the anchors of all slots
    for (int s = 0; s < S; ++s) {
        int32_t* out_idx = m.out_partner + (static_cast<size_t>(row) * S + s) * K;
        float* out_sc = m.out_partner_score + (static_cast<size_t>(row) * S + s) * K;
        const bool live = taken_s[s] >= 0;
        if (live) {
            SelectArgs a = m.base;
            a.mode = kPartnerOnly;
            a.plan = m.plan_partner;
            a.partner_base = slot_ptr(m.base.partner_base, static_cast<size_t>(s) * 2 * kD * esz);
            a.partner_router_query = slot_ptr(m.base.partner_base, (static_cast<size_t>(s) * 2 * kD + kD) * esz);
            a.prq_stride = m.base.pbase_stride;
            a.partner_anchor_cache = slot_ptr(m.base.partner_anchor_cache, s * m.pac_slot);
            a.partner_keys = slot_ptr(m.base.partner_keys, s * m.keys_slot);
            a.partner_mean = slot_ptr(m.base.partner_mean, s * m.stats_slot);
            a.partner_std = slot_ptr(m.base.partner_std, s * m.stats_slot);
            a.partner_gamma = slot_ptr(m.base.partner_gamma, s * m.gamma_slot);
            a.partner_bias = slot_ptr(m.base.partner_bias, s * m.bias_slot);
            a.anchor_index_in = taken_s + s - row;           // [row] == taken_s[s]
            a.exclude_list = taken_s - static_cast<ptrdiff_t>(row) * S;
            a.exclude_count = S;
            a.out_partner = out_idx - static_cast<ptrdiff_t>(row) * K;
            a.out_partner_score = out_sc - static_cast<ptrdiff_t>(row) * K;
            select_row<kDt, false, true>(a, row, smem, smem_u32(&call_bars[4 * (S + s)]));
        }
        __syncthreads();
        if (tid < K) {                                       // the threads that stored the slot's results
            if (!live || !(out_sc[tid] > kNegInf)) { out_idx[tid] = 0; out_sc[tid] = kNegInf; }
        }
        __syncthreads();
    }
}

// ---- whole-sequence (prefill) selection: a tile of consecutive positions per CTA
//
// Query row (b, t) of a whole-sequence pass sees the same block statistics as its neighbours (the
// complete blocks at t) and a local window that overlaps theirs in all but one row.  One CTA
// therefore serves a tile of consecutive positions of one sequence: the statistics of both
// streams and the union of the tile's local windows are staged in shared memory once, then every
// warp takes the tile's queries one at a time and walks the whole chain for its query on its own
// — block scores, local scores, block picking, remote scores (read where the blocks lie, from
// L2), anchor, partner queries, partner scores, top-K — with warp-level synchronisation only.
// The arithmetic is the per-row kernel's own (the same device functions), so indices and scores
// are bit-identical to relation_select_kernel's.
// CTAs of kTileWarps warps serve one, two or four positions per warp (tile_shape).

// ---- warp-per-query primitives (caches, statistics and queries in one dtype kDt: 16 bits, in the decode form fp32 too).
// The arithmetic is the canonical one: every sum below is a sum of the per-row kernel with its operands possibly
// swapped, so scores are bit-identical.  A row is eight chunks of 16 bytes (fp32: 32), lane = 8 rq + chunk: one load
// instruction of a warp covers four whole rows (512 contiguous bytes of a window, of a block's statistics or of a picked
// block in the key cache), a lane keeps only its chunk of the query, and the eight chunk sums of a row meet in a
// butterfly whose level l adds what the per-row kernel's tree adds at level l.  A lane that owned a whole row needed the 64-wide query in
// registers (128 per thread, 16 warps per SM), and remote rows had to pass through shared memory to be read that
// way: 96 cycles of the SM's shared-memory pipe for 32 rows against 39 here.
// Whole-sequence selection of 8 x 4096 rows (384 candidates, 64 blocks): 466 -> 341 us; 16 x 2048 rows of four slots:
// 1233 -> 955 us.  Issue slots 56 -> 71 % taken (69 % since anchor queries stay in 16 bits, below, with 8 % fewer instructions).
constexpr uint32_t kRow = 2 * kD;

// A row in kDt, and a lane's eighth of it: 16 bytes, in single precision (the decode form alone) 32.
template <int kDt> constexpr uint32_t kRowOf = kDt == RLM_F32 ? 4 * kD : kRow;
struct WideChunk { uint4 lo, hi; };
template <int kDt> struct RowChunk { using type = uint4; };
template <> struct RowChunk<RLM_F32> { using type = WideChunk; };
template <int kDt> using Chunk = typename RowChunk<kDt>::type;

template <int kDt>
__device__ __forceinline__ Chunk<kDt> load_chunk(const unsigned char* p) {
    if constexpr (kDt == RLM_F32) return {reinterpret_cast<const uint4*>(p)[0], reinterpret_cast<const uint4*>(p)[1]};
    else return *reinterpret_cast<const uint4*>(p);
}

// Two values of the 16-bit type kDt, from fp32 (exact).
template <int kDt>
__device__ __forceinline__ uint32_t pack_exact(float lo, float hi) {
    if (kDt == RLM_BF16) return (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xffff0000u);
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// This lane's chunk of a query, every element twice: operands of the two-wide fma over two rows.
struct QueryChunk { float2 v[8]; };

__device__ __forceinline__ void load_query_chunk(const float* query, QueryChunk& q) {
    const float* src = query + 8 * (threadIdx.x & 7);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(src + 4 * h);
        q.v[4 * h + 0] = make_float2(x.x, x.x);
        q.v[4 * h + 1] = make_float2(x.y, x.y);
        q.v[4 * h + 2] = make_float2(x.z, x.z);
        q.v[4 * h + 3] = make_float2(x.w, x.w);
    }
}

__device__ __forceinline__ QueryChunk magnitude(const QueryChunk& q) {
    QueryChunk m;
#pragma unroll
    for (int e = 0; e < 8; ++e) m.v[e] = make_float2(fabsf(q.v[e].x), fabsf(q.v[e].y));
    return m;
}

// The chunk of a query whose values are kDt's own (the anchor stream's: a partner query is a sum, rounded to fp32), as
// they lie: the mixed-precision fma takes both factors in 16 bits, widens them exactly and rounds once, the same sums
// as of widened rows in two thirds of the instructions (16 instead of 24 for two rows' chunks; 135 -> 124 million
// for 4 x 4096 rows of a whole-sequence launch, 192 -> 174 us under the profiler).  A multi-anchor pass, us: 16 x 2048 rows of four slots, four layers 11 440 -> 11 270,
// 3 x 1056 rows of two slots, two layers 260 -> 256.
template <int kDt>
struct NarrowChunk { uint32_t v[4]; };

template <int kDt>
__device__ __forceinline__ void load_query_chunk(const float* query, NarrowChunk<kDt>& q) {
    const float* src = query + 8 * (threadIdx.x & 7);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(src + 4 * h);
        q.v[2 * h] = pack_exact<kDt>(x.x, x.y);
        q.v[2 * h + 1] = pack_exact<kDt>(x.z, x.w);
    }
}

template <int kDt>
__device__ __forceinline__ NarrowChunk<kDt> magnitude(const NarrowChunk<kDt>& q) {
    NarrowChunk<kDt> m;
#pragma unroll
    for (int e = 0; e < 4; ++e) m.v[e] = q.v[e] & 0x7fff7fffu;
    return m;
}

// acc + the lower (upper) halves' product, rounded once
template <int kDt>
__device__ __forceinline__ float fma_lower(uint32_t a, uint32_t b, float acc) {
    float d;
    if (kDt == RLM_BF16)
        asm("{.reg .b16 x, y, u, v; mov.b32 {x, y}, %1; mov.b32 {u, v}, %2; fma.rn.f32.bf16 %0, x, u, %3;}" : "=f"(d) : "r"(a), "r"(b), "f"(acc));
    else
        asm("{.reg .b16 x, y, u, v; mov.b32 {x, y}, %1; mov.b32 {u, v}, %2; fma.rn.f32.f16 %0, x, u, %3;}" : "=f"(d) : "r"(a), "r"(b), "f"(acc));
    return d;
}
template <int kDt>
__device__ __forceinline__ float fma_upper(uint32_t a, uint32_t b, float acc) {
    float d;
    if (kDt == RLM_BF16)
        asm("{.reg .b16 x, y, u, v; mov.b32 {x, y}, %1; mov.b32 {u, v}, %2; fma.rn.f32.bf16 %0, y, v, %3;}" : "=f"(d) : "r"(a), "r"(b), "f"(acc));
    else
        asm("{.reg .b16 x, y, u, v; mov.b32 {x, y}, %1; mov.b32 {u, v}, %2; fma.rn.f32.f16 %0, y, v, %3;}" : "=f"(d) : "r"(a), "r"(b), "f"(acc));
    return d;
}

// Element pair i of the chunks of two rows, (lower halves, upper halves), widened to fp32 (exact).
template <int kDt>
__device__ __forceinline__ void widen_pair(uint32_t a, uint32_t b, float2& lower, float2& upper) {
    if (kDt == RLM_BF16) {
        lower = make_float2(__uint_as_float(a << 16), __uint_as_float(b << 16));
        upper = make_float2(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u));
    } else {
        const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&a)), y = __half22float2(*reinterpret_cast<const __half2*>(&b));
        lower = make_float2(x.x, y.x);
        upper = make_float2(x.y, y.y);
    }
}

// seg8 of this lane's chunk for two rows
template <int kDt>
__device__ __forceinline__ float2 seg_pair(const Chunk<kDt> w0, const Chunk<kDt> w1, const QueryChunk& q) {
    if constexpr (kDt == RLM_F32) {
        const uint32_t a[8] = {w0.lo.x, w0.lo.y, w0.lo.z, w0.lo.w, w0.hi.x, w0.hi.y, w0.hi.z, w0.hi.w};
        const uint32_t b[8] = {w1.lo.x, w1.lo.y, w1.lo.z, w1.lo.w, w1.hi.x, w1.hi.y, w1.hi.z, w1.hi.w};
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc = __ffma2_rn(make_float2(__uint_as_float(a[i]), __uint_as_float(b[i])), q.v[i], acc);
        return acc;
    } else {
    const uint32_t a[4] = {w0.x, w0.y, w0.z, w0.w}, b[4] = {w1.x, w1.y, w1.z, w1.w};
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 lower, upper;
        widen_pair<kDt>(a[i], b[i], lower, upper);
        acc = __ffma2_rn(lower, q.v[2 * i], acc);
        acc = __ffma2_rn(upper, q.v[2 * i + 1], acc);
    }
    return acc;
    }
}

template <int kDt>
__device__ __forceinline__ float2 seg_pair(const uint4 w0, const uint4 w1, const NarrowChunk<kDt>& q) {
    const uint32_t a[4] = {w0.x, w0.y, w0.z, w0.w}, b[4] = {w1.x, w1.y, w1.z, w1.w};
    float x = 0.0f, y = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x = fma_lower<kDt>(a[i], q.v[i], x);
        y = fma_lower<kDt>(b[i], q.v[i], y);
        x = fma_upper<kDt>(a[i], q.v[i], x);
        y = fma_upper<kDt>(b[i], q.v[i], y);
    }
    return make_float2(x, y);
}

// One level of the butterfly over the chunk lanes: of kN values (a row each) a lane keeps those whose index has the
// parity of its lane bit, adds the partner's halves of them and hands over its own halves of the others.
template <int kN, int kXor>
__device__ __forceinline__ void fold_level(const float (&s)[kN], float (&out)[kN / 2]) {
    const bool odd = threadIdx.x & kXor;
#pragma unroll
    for (int j = 0; j < kN / 2; ++j) {
        const float keep = odd ? s[2 * j + 1] : s[2 * j], give = odd ? s[2 * j] : s[2 * j + 1];
        out[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, kXor));
    }
}

// Chunk sums of rows load(0) .. load(kN - 1) (row i: rows 4 i + rq of a pass), two rows at a time.
template <int kDt, int kN, typename Load, typename Query>
__device__ __forceinline__ void chunk_sums(const Load& load, const Query& q, float (&s)[kN]) {
    constexpr int kStep = kN < 4 ? kN : 4;
#pragma unroll
    for (int h = 0; h < kN; h += kStep) {
        Chunk<kDt> w[kStep];
#pragma unroll
        for (int i = 0; i < kStep; ++i) w[i] = load(h + i);
#pragma unroll
        for (int i = 0; i < kStep; i += 2) {
            const float2 p = seg_pair<kDt>(w[i], w[i + 1], q);
            s[h + i] = p.x;
            s[h + i + 1] = p.y;
        }
    }
}

// Score of the row that this lane owns after the butterfly: row 4 (chunk mod kN) + rq of a pass of 4 kN rows (with
// fewer than eight rows per lane group, lanes own rows in common).  A pass of 32 rows costs the least per row; one of
// 16 or 8 ends sooner, where warps are idle.
template <int kDt, int kN, typename Load, typename Query>
__device__ __forceinline__ float pass_score(const Load& load, const Query& q) {
    float s[kN], total;
    chunk_sums<kDt, kN>(load, q, s);
    if constexpr (kN == 8) {
        float v[4], u[2], t[1];
        fold_level<8, 1>(s, v);
        fold_level<4, 2>(v, u);
        fold_level<2, 4>(u, t);
        total = t[0];
    } else if constexpr (kN == 4) {
        float v[2], u[1];
        fold_level<4, 1>(s, v);
        fold_level<2, 2>(v, u);
        total = __fadd_rn(u[0], __shfl_xor_sync(0xffffffffu, u[0], 4));
    } else {
        float v[1];
        fold_level<2, 1>(s, v);
        const float u = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], 2));
        total = __fadd_rn(u, __shfl_xor_sync(0xffffffffu, u, 4));
    }
    return __fmul_rn(total, 0.125f);
}

// Further excluded positions of a query (the anchors of a multi-anchor row's slots; -1 = none).
struct ExclRegs { int v[kMaxExclude]; int n; };

template <bool kExcl>
__device__ __forceinline__ bool not_excluded(int pos, const ExclRegs* ex) {
    bool keep = true;
    if (kExcl) {                       // unused entries are -1, which no position equals
#pragma unroll
        for (int x = 0; x < kMaxExclude / 2; ++x) keep = keep && pos != ex->v[x];
        if (ex->n > kMaxExclude / 2) {
#pragma unroll
            for (int x = kMaxExclude / 2; x < kMaxExclude; ++x) keep = keep && pos != ex->v[x];
        }
    }
    return keep;
}

// Best (score, lowest position on ties) of the warp into the running best.
__device__ __forceinline__ void fold_best(uint32_t my_key, int my_pos, uint32_t& best_key, int& best_pos) {
    warp_argmax_key(my_key, my_pos);
    if (my_pos != 0x7fffffff &&
        (my_key > best_key || best_pos == 0x7fffffff || (my_key == best_key && my_pos < best_pos))) {
        best_key = my_key;
        best_pos = my_pos;
    }
}

__device__ __forceinline__ void keep_best(bool valid, float score, int pos, uint32_t& my_key, int& my_pos) {
    const uint32_t key = float_key(score);
    if (valid && (key > my_key || my_pos == 0x7fffffff || (key == my_key && pos < my_pos))) {
        my_key = key;
        my_pos = pos;
    }
}

// The passes first, first + step, ... of a score function are this warp's (all of them by default).

// The local window, staged in shared memory: row r is position pos0 + r; rows below first_valid are none (and
// not staged).  Scores go to cand[slot0 + r], or, without cand, into the running
// best (kBoth: to both).
template <int kDt, bool kExcl = false, bool kBoth = false, int kN = 8, typename Query>
__device__ __forceinline__ void score_window_warp(const unsigned char* rows, int n_rows, int first_valid, int pos0, int exclude,
                                                  const Query& q, float* cand, int slot0, uint32_t& best_key,
                                                  int& best_pos, const ExclRegs* ex = nullptr, int first = 0, int step = 1) {
    const int lane = threadIdx.x & 31, chunk = lane & 7, rq = lane >> 3;
    uint32_t my_key = 0;
    int my_pos = 0x7fffffff;
    const unsigned char* mine = rows + kRowOf<kDt> / 8 * chunk;
    for (int base = 4 * kN * first; base < n_rows; base += 4 * kN * step) {
        float sc;
        if (base >= first_valid && base + 4 * kN <= n_rows) {
            const unsigned char* src = mine + (base + rq) * static_cast<int>(kRowOf<kDt>);
            sc = pass_score<kDt, kN>([&](int i) { return load_chunk<kDt>(src + i * static_cast<int>(4 * kRowOf<kDt>)); }, q);
        } else {
            // the ragged ends read a staged row in place of each missing one
            sc = pass_score<kDt, kN>([&](int i) {
                const int r = min(max(base + 4 * i + rq, first_valid), n_rows - 1);
                return load_chunk<kDt>(mine + r * static_cast<int>(kRowOf<kDt>));
            }, q);
        }
        const int r = base + 4 * (chunk & (kN - 1)) + rq, pos = pos0 + r;
        const bool valid = r < n_rows && r >= first_valid && pos != exclude && not_excluded<kExcl>(pos, ex);
        sc = valid ? sc : kNegInf;
        if (kBoth || cand)
            if (r < n_rows) cand[slot0 + r] = sc;
        if (kBoth || !cand) keep_best(valid, sc, pos, my_key, my_pos);
    }
    if (kBoth || !cand) fold_best(my_key, my_pos, best_key, best_pos);
}

// The picked remote blocks (sel: block, picked, rows), scored where they lie in the key cache.
template <int kDt, bool kExcl = false, bool kBoth = false, int kN = 8, typename Query>
__device__ __forceinline__ void score_remote_warp(const unsigned char* keys, int n_rows, const int* sel, int bs,
                                                  int bs_shift, int exclude, const Query& q, float* cand, int slot0,
                                                  uint32_t& best_key, int& best_pos, const ExclRegs* ex = nullptr,
                                                  int first = 0, int step = 1) {
    const int lane = threadIdx.x & 31, chunk = lane & 7, rq = lane >> 3;
    uint32_t my_key = 0;
    int my_pos = 0x7fffffff;
    const unsigned char* mine = keys + kRowOf<kDt> / 8 * chunk;
    for (int base = 4 * kN * first; base < n_rows; base += 4 * kN * step) {
        const int r = base + 4 * (chunk & (kN - 1)) + rq;
        int pos;                                         // position of row r, or -1
        float sc;
        if (bs_shift >= (kN == 8 ? 5 : kN == 4 ? 4 : 3)) {
            // the pass lies in one picked block: rows 4 i + rq are 512 bytes apart
            const int rank = base >> bs_shift, o0 = base - (rank << bs_shift);
            const int start = sel[3 * rank] * bs + o0, lim = sel[3 * rank + 2] - o0;
            const unsigned char* src = mine + static_cast<size_t>(start + rq) * kRowOf<kDt>;
            // rows past `lim` are read too (they lie inside the block, hence inside the cache) and ignored
            sc = pass_score<kDt, kN>([&](int i) { return load_chunk<kDt>(src + i * static_cast<int>(4 * kRowOf<kDt>)); }, q);
            pos = r - base < lim ? start + (r - base) : -1;
        } else {
            auto row_pos = [&](int row) -> int {
                if (row >= n_rows) return -1;
                const int rank = bs_shift >= 0 ? row >> bs_shift : row / bs, o = row - rank * bs;
                return o < sel[3 * rank + 2] ? sel[3 * rank] * bs + o : -1;
            };
            sc = pass_score<kDt, kN>([&](int i) {
                const int p = row_pos(base + 4 * i + rq);
                return p >= 0 ? load_chunk<kDt>(mine + static_cast<size_t>(p) * kRowOf<kDt>) : Chunk<kDt>{};
            }, q);
            pos = row_pos(r);
        }
        const bool valid = pos >= 0 && pos != exclude && not_excluded<kExcl>(pos, ex);
        sc = valid ? sc : kNegInf;
        if (kBoth || cand)
            if (r < n_rows) cand[slot0 + r] = sc;
        if (kBoth || !cand) keep_best(valid, sc, pos, my_key, my_pos);
    }
    if (kBoth || !cand) fold_best(my_key, my_pos, best_key, best_pos);
}

// score_blocks for one warp, 32 blocks a pass: chunks 2 h and 2 h + 1 of a block's statistics are head h, so the
// first butterfly level completes a head's sums; a 4 x 4 transpose between the head lanes then leaves every lane
// with the four heads of one block.  out[n] for the first n_complete blocks, -inf up to the next multiple of four
// of nb.
template <int kDt, typename Query>
__device__ __forceinline__ void score_blocks_warp(const unsigned char* mean, const unsigned char* stdv, int nb, int n_complete,
                                                  int bs, int t, int ls, int strict, int buckets, const Query& q,
                                                  const float* sp4, const float* bias, float* out, int first = 0, int step = 1) {
    const int lane = threadIdx.x & 31, chunk = lane & 7, rq = lane >> 3;
    if (first == 0)
        for (int n = n_complete + lane; n < ((nb + 3) & ~3); n += 32) out[n] = kNegInf;
    const auto qa = magnitude(q);
    const float sp = sp4[chunk >> 1];
    const bool x2 = lane & 2, x4 = lane & 4;
    for (int base = 32 * first; base < n_complete; base += 32 * step) {
        float sums[8], md[4], sd[4];
        const auto at = [&](int i) { return static_cast<uint32_t>(min(base + 4 * i + rq, n_complete - 1)) * kRowOf<kDt> + kRowOf<kDt> / 8 * chunk; };
        chunk_sums<kDt, 8>([&](int i) { return load_chunk<kDt>(mean + at(i)); }, q, sums);
        fold_level<8, 1>(sums, md);
        chunk_sums<kDt, 8>([&](int i) { return load_chunk<kDt>(stdv + at(i)); }, qa, sums);
        fold_level<8, 1>(sums, sd);
        // v[j]: head (chunk >> 1) of block 4 (2 j + (chunk & 1)) + rq
        float v[4], w[2][2], sh[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = __fmul_rn(__fadd_rn(md[j], __fmul_rn(sp, sd[j])), 0.25f);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float got = __shfl_xor_sync(0xffffffffu, x2 ? v[2 * j] : v[2 * j + 1], 2), own = x2 ? v[2 * j + 1] : v[2 * j];
            w[j][0] = x2 ? got : own;
            w[j][1] = x2 ? own : got;
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const float got = __shfl_xor_sync(0xffffffffu, x4 ? w[0][x] : w[1][x], 4), own = x4 ? w[1][x] : w[0][x];
            sh[x] = x4 ? got : own;
            sh[2 + x] = x4 ? own : got;
        }
        const int n = base + 4 * chunk + rq;
        if (n >= n_complete) continue;                   // no lane-collective operation follows in the pass
        const int end = (n + 1) * bs - 1;
        int dist = t - end;
        if (dist < 0) dist = 0;
        int bucket = 31 - __clz(dist + 1);
        if (bucket > buckets - 1) bucket = buckets - 1;
#pragma unroll
        for (int h = 0; h < 4; ++h) sh[h] = __fadd_rn(sh[h], bias[h * buckets + bucket]);
        const float mx = fmaxf(fmaxf(sh[0], sh[1]), fmaxf(sh[2], sh[3]));
        const float e01 = __fadd_rn(canon_exp(__fsub_rn(sh[0], mx)), canon_exp(__fsub_rn(sh[1], mx)));
        const float e23 = __fadd_rn(canon_exp(__fsub_rn(sh[2], mx)), canon_exp(__fsub_rn(sh[3], mx)));
        const float acc = __fadd_rn(mx, canon_log(__fadd_rn(e01, e23)));
        out[n] = (!strict || end < ls) ? acc : kNegInf;
    }
}

// Scores of eight blocks, first .. first + 7: a lane pair has one head of one block, and the heads of a block meet in
// two more exchanges.  Half the time of a pass of 32, for few blocks and warps to spare.  `sp` and `shift`: this lane's
// head's softplus(gamma) and its bias at the block's distance (block_shift).
__device__ __forceinline__ int lane_block(int first) { return first + 4 * (threadIdx.x & 1) + ((threadIdx.x & 31) >> 3); }

__device__ __forceinline__ float block_shift(const void* bias, int block, int bs, int t, int buckets, int dtype) {
    int bucket = 31 - __clz(max(t - ((block + 1) * bs - 1), 0) + 1);
    if (bucket > buckets - 1) bucket = buckets - 1;
    return load_scalar(bias, ((threadIdx.x & 7) >> 1) * buckets + bucket, dtype);
}

template <int kDt>
__device__ __forceinline__ void score_eight_blocks(const unsigned char* mean, const unsigned char* stdv, int first, int n_complete,
                                                   int bs, int ls, int strict, const QueryChunk& q, float sp, float shift,
                                                   float* out) {
    const int lane = threadIdx.x & 31, chunk = lane & 7, rq = lane >> 3;
    const auto qa = magnitude(q);
    float sums[2], md[1], sd[1];
    const auto at = [&](int i) { return static_cast<uint32_t>(min(first + 4 * i + rq, n_complete - 1)) * kRowOf<kDt> + kRowOf<kDt> / 8 * chunk; };
    chunk_sums<kDt, 2>([&](int i) { return load_chunk<kDt>(mean + at(i)); }, q, sums);
    fold_level<2, 1>(sums, md);
    chunk_sums<kDt, 2>([&](int i) { return load_chunk<kDt>(stdv + at(i)); }, qa, sums);
    fold_level<2, 1>(sums, sd);
    const float sh = __fadd_rn(__fmul_rn(__fadd_rn(md[0], __fmul_rn(sp, sd[0])), 0.25f), shift);
    float mx = fmaxf(sh, __shfl_xor_sync(0xffffffffu, sh, 2));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    float e = canon_exp(__fsub_rn(sh, mx));
    e = __fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, 2));
    e = __fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, 4));
    const int n = lane_block(first);
    if (n < n_complete) out[n] = (!strict || (n + 1) * bs - 1 < ls) ? __fadd_rn(mx, canon_log(e)) : kNegInf;
}

// The choices of pick_blocks among up to 32 blocks, a block a lane: lane r gets the r-th, or -1.
__device__ __forceinline__ int pick_small(const float* scores, int nb, int top) {
    const int lane = threadIdx.x & 31;
    const float v = lane < nb ? scores[lane] : kNegInf;
    uint32_t key = v > -1.0e30f ? float_key(v + 0.0f) : 0u;
    int picked = -1;
    for (int r = 0; r < top; ++r) {
        const uint32_t best = __reduce_max_sync(0xffffffffu, key);
        if (best == 0u) break;
        const int n = __ffs(__ballot_sync(0xffffffffu, key == best)) - 1;
        picked = lane == r ? n : picked;
        key = lane == n ? 0u : key;
    }
    return picked;
}

// The list entry (block, picked, rows) of a choice.
__device__ __forceinline__ void write_pick(int* entry, int picked, int bs, int ls) {
    entry[0] = max(picked, 0);
    entry[1] = picked >= 0;
    entry[2] = picked < 0 ? 0 : min(max(ls - picked * bs, 0), bs);
}

// Pass `first` of the picked rows with the choices in registers (lane r: the r-th) and a pass inside one block.
template <int kDt, int kN>
__device__ __forceinline__ void score_picked_pass(const unsigned char* keys, int first, int picked, int bs, int bs_shift, int ls,
                                                  int exclude, const QueryChunk& q, float* cand, uint32_t& best_key, int& best_pos) {
    const int lane = threadIdx.x & 31, chunk = lane & 7, rq = lane >> 3, base = 4 * kN * first;
    const int rank = base >> bs_shift, o0 = base - (rank << bs_shift), block = __shfl_sync(0xffffffffu, picked, rank);
    const int start = max(block, 0) * bs + o0, lim = block < 0 ? 0 : min(max(ls - block * bs, 0), bs) - o0;
    const unsigned char* src = keys + static_cast<size_t>(start + rq) * kRowOf<kDt> + kRowOf<kDt> / 8 * chunk;
    // rows past `lim` are read too (they lie inside the block, hence inside the cache) and ignored
    float sc = pass_score<kDt, kN>([&](int i) { return load_chunk<kDt>(src + i * static_cast<int>(4 * kRowOf<kDt>)); }, q);
    const int o = 4 * (chunk & (kN - 1)) + rq, pos = start + o;
    const bool valid = o < lim && pos != exclude;
    sc = valid ? sc : kNegInf;
    cand[base + o] = sc;
    uint32_t my_key = 0;
    int my_pos = 0x7fffffff;
    keep_best(valid, sc, pos, my_key, my_pos);
    fold_best(my_key, my_pos, best_key, best_pos);
}

// pick_blocks for one warp and up to 128 blocks: `top` rounds of (largest score, lowest block on
// ties) through two redux instructions each, instead of ranking every block against all others.
__device__ __forceinline__ void pick_blocks_warp(const float* scores, int nb, int top, int bs, int ls, int* sel) {
    const int lane = threadIdx.x & 31;
    if (nb <= 32) {
        const int picked = pick_small(scores, nb, top);
        if (lane < top) write_pick(sel + 3 * lane, picked, bs, ls);
        __syncwarp();
        return;
    }
    uint32_t key[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int n = lane + 32 * i;
        const float v = n < nb ? scores[n] : kNegInf;
        key[i] = v > -1.0e30f ? float_key(v + 0.0f) : 0u;
    }
    for (int r = lane; r < top; r += 32) { sel[3 * r] = 0; sel[3 * r + 1] = 0; sel[3 * r + 2] = 0; }
    __syncwarp();
    for (int r = 0; r < top; ++r) {
        uint32_t mk = key[0];
        int mi = 0;
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (key[i] > mk) { mk = key[i]; mi = i; }
        const uint32_t best = __reduce_max_sync(0xffffffffu, mk);
        if (best == 0u) break;
        const int mine = mk == best ? lane + 32 * mi : 0x7fffffff;
        const int n = __reduce_min_sync(0xffffffffu, mine);
        if (mine == n) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == mi) key[i] = 0u;
            int rows = ls - n * bs;
            rows = rows < 0 ? 0 : (rows > bs ? bs : rows);
            sel[3 * r] = n;
            sel[3 * r + 1] = 1;
            sel[3 * r + 2] = rows;
        }
    }
    __syncwarp();
}

// Exact top-K by one warp through a threshold: the K-th largest of the 32 lane maxima is a lower
// bound of the K-th largest score, so only candidates at or above it can be selected; they are
// compacted (64 words of `scratch`) and ranked exactly, higher score first and equal scores by the
// earlier slot, as topk_tournament orders them.  Returns false, with nothing written, when fewer
// than K lanes hold a finite score or more than 32 candidates pass (many equal scores): the
// caller then runs the tournament.
template <int kN>
__device__ __forceinline__ bool topk_filter(const float* cand, int cap4, int K, int L, int t, int bs, int bs_shift,
                                            const int* sel, uint32_t* scratch, int32_t* out_pos, float* out_score) {
    const int lane = threadIdx.x & 31;
    uint32_t k[kN], active = 0;
#pragma unroll
    for (int i = 0; i < kN; ++i) {
        const int slot = 32 * i + lane;
        k[i] = slot < cap4 ? float_key(cand[slot] + 0.0f) : 0u;
        active = max(active, k[i]);
    }
    uint32_t tau = 0;
    for (int r = 0; r < K; ++r) {
        tau = __reduce_max_sync(0xffffffffu, active);
        const int w = __ffs(__ballot_sync(0xffffffffu, active == tau)) - 1;
        if (lane == w) active = 0u;
    }
    if (tau <= float_key(kNegInf)) return false;
    int count = 0;
#pragma unroll
    for (int i = 0; i < kN; ++i) {
        const bool pass = k[i] >= tau;
        const unsigned b = __ballot_sync(0xffffffffu, pass);
        const int at = count + __popc(b & ((1u << lane) - 1u));
        if (pass && at < 32) {
            scratch[2 * at] = k[i];
            scratch[2 * at + 1] = static_cast<uint32_t>(32 * i + lane);
        }
        count += __popc(b);
    }
    if (count > 32) return false;
    __syncwarp();
    if (lane < count) {
        const uint32_t key = scratch[2 * lane], slot = scratch[2 * lane + 1];
        int rank = 0;
        for (int j = 0; j < count; ++j) {
            const uint32_t kj = scratch[2 * j], sj = scratch[2 * j + 1];
            rank += (kj > key) || (kj == key && sj < slot);
        }
        if (rank < K) {
            const float sc = cand[slot];
            const int cs = static_cast<int>(slot);
            int pos;
            if (!(sc > kNegInf)) pos = t - L + 1;
            else if (cs < L) pos = t - L + 1 + cs;
            else { const int rr = bs_shift >= 0 ? (cs - L) >> bs_shift : (cs - L) / bs; pos = sel[3 * rr] * bs + (cs - L - rr * bs); }
            out_pos[rank] = pos;
            out_score[rank] = sc;
        }
    }
    __syncwarp();
    return true;
}

// Exact top-K of up to 512 candidate slots by one warp.
__device__ __forceinline__ void topk_warp(const float* cand, int cap4, int K, int L, int t, int bs, int bs_shift, const int* sel,
                                          uint32_t* scratch, int32_t* out_pos, float* out_score) {
    if (cap4 <= 128) {
        if (!topk_filter<4>(cand, cap4, K, L, t, bs, bs_shift, sel, scratch, out_pos, out_score))
            topk_tournament<4>(cand, cap4, K, L, t, bs, bs_shift, sel, out_pos, out_score);
    } else if (cap4 <= 256) {
        if (!topk_filter<8>(cand, cap4, K, L, t, bs, bs_shift, sel, scratch, out_pos, out_score))
            topk_tournament<8>(cand, cap4, K, L, t, bs, bs_shift, sel, out_pos, out_score);
    } else {
        if (!topk_filter<16>(cand, cap4, K, L, t, bs, bs_shift, sel, scratch, out_pos, out_score))
            topk_tournament<16>(cand, cap4, K, L, t, bs, bs_shift, sel, out_pos, out_score);
    }
}

// How many of 4 n_groups keys come before `mine`, number `index` of them: the larger, and the equal ones of lower
// number; mine > 0.  Four counters, so that the additions do not wait for one another.
template <int kUnroll>
__device__ __forceinline__ int rank_among(const uint32_t* keys, int n_groups, uint32_t mine, int index) {
    const uint32_t before = mine - 1u;                       // k > before: k >= mine
    const int own = index >> 2, at = index & 3;
    const uint4 k0 = *reinterpret_cast<const uint4*>(keys + 4 * own);
    int r0 = k0.x == mine && at > 0, r1 = k0.y == mine && at > 1, r2 = k0.z == mine && at > 2, r3 = 0;
#pragma unroll kUnroll
    for (int g = 0; g < n_groups; ++g) {
        const uint4 k = *reinterpret_cast<const uint4*>(keys + 4 * g);
        const uint32_t bar = g < own ? before : mine;
        if (k.x > bar) ++r0;
        if (k.y > bar) ++r1;
        if (k.z > bar) ++r2;
        if (k.w > bar) ++r3;
    }
    return (r0 + r1) + (r2 + r3);
}

// ---- the decode form in one dtype: a query row by a CTA of eight warps
//
// A row's time is a chain of dependent phases, so what counts is their number and length, not their work.  Here a
// phase is a pass of 32 rows or blocks by a warp (the primitives above: a handful of loads, 64 multiply-adds a lane, a
// three-step butterfly): complete blocks and local window side by side, then every warp that has picked rows to score
// ranks the block scores for itself (top rounds of two redux instructions) and scores its passes, all warps merge the
// eight warps' bests, add the anchor's partner-query row and do the same for the partners; the top K come from ranking
// every candidate against all others by the whole CTA.  Half of a cold phase is instruction fetch (a pass of blocks
// takes 2300 cycles where its arithmetic needs some 900), so both streams run through one copy of the code.
// In fp32 a lane's eighth of a row is 32 bytes, and whole caches fit where 512 bytes a position and 1024 a block leave some
// 2.5 KB of 220 (384 positions in 12 blocks, 344 in 43): 9.4 -> 6.2 us at one row of 128 positions, 10.5 -> 9.1 at 512 (window
// alone), against select_row.
// kResident: both key caches of the sequence in shared memory (requested before the dependency wait), else the window
// there and the picked rows from L2.
// kCtaTop: the top K of 257 to 512 candidates by the CTA, as in select_row, not by a warp (fp32, whose scores that are NaN
// then rank as in launches of more rows).  A build of its own: without the warp's top K the other one's code is the slower,
// whether a launch comes there or not (us a step of batch 7, d 768, 5 layers 272.8 -> 275.7).
template <int kDt, bool kResident, bool kCtaTop = false>
__global__ void __launch_bounds__(kThreads, kResident ? 1 : 2) relation_select_decode_kernel(const SelectArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t best_key_s[kWarps], short_list[64];
    __shared__ __align__(16) int best_pos_s[kWarps], sel_s[kWarps * 3 * kDecodeTop];
    __shared__ float softplus_s[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = blockIdx.x, buckets4 = 4 * a.buckets;
    const Plan& p = a.plan;
    const uint32_t bar_a = smem_u32(smem + p.bars), bar_p = bar_a + 8;
    // The caches, statistics and the position were written before the previous kernel of the stream started, so
    // everything up to the bulk-copy requests may run while that kernel (which makes the queries) is still executing.
    const int t = static_cast<int>(*a.position);
    const int nb = a.n_blocks, bs = a.block_size, L = a.local_window, top = a.top_blocks;
    const int bs_shift = (bs & (bs - 1)) == 0 ? 31 - __clz(bs) : -1;
    const int ls = max(t - L + 1, 0), first_local = ls - (t - L + 1), n_complete = max(min((t + 1) / bs, nb), 0);
    const size_t seq_keys = static_cast<size_t>(row) * a.max_t * kRowOf<kDt>, seq_stats = static_cast<size_t>(row) * nb * kRowOf<kDt>;
    const int cap = L + top * bs, cap4 = (cap + 3) & ~3;
    const bool bad_position = t < 0 || t >= a.max_t;
    if (tid == 0 && !bad_position) {
        mbar_init(bar_a, 1);
        mbar_init(bar_p, 1);
        fence_barrier_init();
        const uint32_t sbytes = top > 0 ? n_complete * kRowOf<kDt> : 0u;
        const uint32_t lbytes = (kResident ? t + 1 : t - ls + 1) * kRowOf<kDt>;
        const size_t loff = seq_keys + (kResident ? 0 : static_cast<size_t>(ls) * kRowOf<kDt>);
        const uint32_t ldst = kResident ? 0u : first_local * kRowOf<kDt>;
        const auto request = [&](const void* mean, const void* stdv, const void* keys, int mean_at, int std_at, int keys_at,
                                 uint32_t bar) {
            mbar_expect_tx(bar, 2 * sbytes + lbytes);
            if (sbytes) {
                bulk_g2s(smem_u32(smem + mean_at), static_cast<const char*>(mean) + seq_stats, sbytes, bar);
                bulk_g2s(smem_u32(smem + std_at), static_cast<const char*>(stdv) + seq_stats, sbytes, bar);
            }
            bulk_g2s(smem_u32(smem + keys_at) + ldst, static_cast<const char*>(keys) + loff, lbytes, bar);
        };
        request(a.anchor_mean, a.anchor_std, a.anchor_keys, p.a_mean, p.a_std, p.a_local, bar_a);
        request(a.partner_mean, a.partner_std, a.partner_keys, p.p_mean, p.p_std, p.p_local, bar_p);
    }
    float* queries = reinterpret_cast<float*>(smem + p.queries);                 // aq | arq | pq | prq
    float* bias_a = reinterpret_cast<float*>(smem + p.params), *bias_p = bias_a + buckets4;
    float* bscore = reinterpret_cast<float*>(smem + p.block_scores);
    float* cand = reinterpret_cast<float*>(smem + p.cand);
    for (int i = tid; i < buckets4; i += kThreads) {
        bias_a[i] = load_scalar(a.anchor_bias, i, a.param_dtype);
        bias_p[i] = load_scalar(a.partner_bias, i, a.param_dtype);
    }
    if (tid < cap4 - cap) cand[cap + tid] = kNegInf;             // padding slots never win a comparison
    const bool few_blocks = n_complete <= 32;
    for (int n = n_complete + tid; n < ((nb + 3) & ~3); n += kThreads) bscore[n] = kNegInf;
    // few blocks: eight to a warp, whose lanes keep their head's parameters for both streams
    float lane_sp[2] = {0.0f, 0.0f}, lane_shift[2] = {0.0f, 0.0f};
    if (few_blocks && !bad_position && 8 * warp < n_complete) {
        const int head = (tid & 7) >> 1, block = lane_block(8 * warp);
        lane_sp[0] = canon_log(__fadd_rn(1.0f, canon_exp(load_scalar(a.anchor_gamma, head, a.param_dtype))));
        lane_sp[1] = canon_log(__fadd_rn(1.0f, canon_exp(load_scalar(a.partner_gamma, head, a.param_dtype))));
        lane_shift[0] = block_shift(a.anchor_bias, block, bs, t, a.buckets, a.param_dtype);
        lane_shift[1] = block_shift(a.partner_bias, block, bs, t, a.buckets, a.param_dtype);
    }
    // parameters that are first used behind the wait, into the constant cache
    asm volatile("" ::"l"(a.anchor_query), "l"(a.anchor_router_query), "l"(a.partner_base), "l"(a.partner_anchor_cache),
                 "l"(a.out_anchor), "l"(a.out_anchor_score), "l"(a.out_partner), "l"(a.out_partner_score), "l"(a.aq_stride),
                 "l"(a.arq_stride), "l"(a.pbase_stride), "r"(a.k_out), "r"(a.strict_valid));
    if (tid >= 32 && tid < 40)
        softplus_s[tid - 32] = canon_log(__fadd_rn(1.0f, canon_exp(load_scalar(tid < 36 ? a.anchor_gamma : a.partner_gamma, tid & 3, a.param_dtype))));
    griddep_sync();
    if (bad_position) {
        if (tid == 0 && a.status) atomicOr(a.status, RLM_DEV_POSITION);
        return;
    }
    queries[tid] = tid < kD       ? load_scalar(a.anchor_query, row * a.aq_stride + tid, kDt)
                   : tid < 2 * kD ? load_scalar(a.anchor_router_query, row * a.arq_stride + tid - kD, kDt)
                                  : load_scalar(a.partner_base, row * a.pbase_stride + tid - 2 * kD, kDt);
    __syncthreads();

    // blocks and window side by side: up to half of the warps walk the passes of blocks
    const int block_warps = top > 0 ? max(1, min(few_blocks ? (n_complete + 7) >> 3 : (n_complete + 31) >> 5, kWarps / 2)) : 0;
    const int picked_rows = top * bs;
    int* sel = sel_s + warp * 3 * kDecodeTop;
    // row r of a window is position t - L + 1 + r (only rows that are staged are read)
    const ptrdiff_t window_offset = kResident ? static_cast<ptrdiff_t>(t - L + 1) * static_cast<ptrdiff_t>(kRowOf<kDt>) : 0;
    int anchor_pos = -1;
    // the anchor's stream, then the partner's: one copy of the code, so that the second finds it in the instruction cache
#pragma unroll 1
    for (int stream = 0; stream < 2; ++stream) {
        const unsigned char* mean = smem + (stream ? p.p_mean : p.a_mean), *stdv = smem + (stream ? p.p_std : p.a_std);
        const unsigned char* staged = smem + (stream ? p.p_local : p.a_local);
        const unsigned char* keys = static_cast<const unsigned char*>(stream ? a.partner_keys : a.anchor_keys) + seq_keys;
        const float* query = queries + 2 * kD * stream;            // exact query | router query
        const bool ok = mbar_wait(stream ? bar_p : bar_a, 0);
        QueryChunk q;
        uint32_t bk = 0;
        int bp = 0x7fffffff;
        if (warp < block_warps) {
            load_query_chunk(query + kD, q);
            if (!few_blocks)
                score_blocks_warp<kDt>(mean, stdv, nb, n_complete, bs, t, ls, a.strict_valid, a.buckets, q, softplus_s + 4 * stream,
                                       stream ? bias_p : bias_a, bscore, warp, block_warps);
            else if (n_complete > 0)
                score_eight_blocks<kDt>(mean, stdv, 8 * warp, n_complete, bs, ls, a.strict_valid, q, stream ? lane_sp[1] : lane_sp[0],
                                        stream ? lane_shift[1] : lane_shift[0], bscore);
            load_query_chunk(query, q);
        } else {
            load_query_chunk(query, q);
            const unsigned char* window = staged + window_offset;
            const int first = warp - block_warps, step = kWarps - block_warps;
            if (L <= 16 * step)
                score_window_warp<kDt, false, true, 4>(window, L, first_local, t - L + 1, anchor_pos, q, cand, 0, bk, bp, nullptr,
                                                       first, step);
            else
                score_window_warp<kDt, false, true>(window, L, first_local, t - L + 1, anchor_pos, q, cand, 0, bk, bp, nullptr,
                                                    first, step);
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0 && a.status) atomicOr(a.status, RLM_DEV_TIMEOUT);
            return;
        }
        const unsigned char* rows = kResident ? staged : keys;
        if (nb <= 32 && bs_shift >= 4 && picked_rows <= 16 * kWarps) {
            // a pass of 8 or 16 rows per warp, each inside one block; the first warp leaves the list for the top K
            const int pass_rows = picked_rows <= 8 * kWarps ? 8 : 16;
            if (pass_rows * warp < picked_rows) {
                const int picked = pick_small(bscore, nb, top);
                if (pass_rows == 8)
                    score_picked_pass<kDt, 2>(rows, warp, picked, bs, bs_shift, ls, anchor_pos, q, cand + L, bk, bp);
                else
                    score_picked_pass<kDt, 4>(rows, warp, picked, bs, bs_shift, ls, anchor_pos, q, cand + L, bk, bp);
                if (warp == 0 && lane < top) write_pick(sel + 3 * lane, picked, bs, ls);
            }
        } else if (32 * warp < picked_rows) {
            if (nb <= 128) pick_blocks_warp(bscore, nb, top, bs, ls, sel);
            else pick_blocks(bscore, nb, top, bs, ls, sel);
            score_remote_warp<kDt, false, true>(rows, picked_rows, sel, bs, bs_shift, anchor_pos, q, cand, L, bk, bp, nullptr, warp,
                                                kWarps);
        }
        if (lane == 0) { best_key_s[warp] = bk; best_pos_s[warp] = bp; }
        __syncthreads();
        if (stream) break;
        // highest score wins; equal scores go to the lowest position (the reference's left-most local arg-max followed
        // by its "equal and earlier" merge rule)
        uint32_t best_key = lane < kWarps ? best_key_s[lane] : 0u;
        anchor_pos = lane < kWarps ? best_pos_s[lane] : 0x7fffffff;
        if (anchor_pos == 0x7fffffff) best_key = 0u;
        warp_argmax_key(best_key, anchor_pos);
        if (anchor_pos == 0x7fffffff) {   // no candidate
            anchor_pos = 0;
            best_key = float_key(kNegInf);
        }
        if (tid < 2 * kD)       // the anchor's contribution to the partner queries
            queries[2 * kD + tid] = __fadd_rn(queries[2 * kD + tid],
                                              load_scalar(a.partner_anchor_cache, (static_cast<size_t>(row) * a.max_t + anchor_pos) * 2 * kD + tid, kDt));
        if (tid == kThreads - 1) {
            a.out_anchor[row] = anchor_pos;
            a.out_anchor_score[row] = key_float(best_key);
        }
        __syncthreads();
    }
    // Exact top-K of the candidate table: output slot k holds the k-th best candidate (higher score first, equal scores
    // by the earlier slot); results without a finite score report -inf and the position of candidate slot 0.
    const int K = a.k_out;
    int32_t* out_pos = a.out_partner + static_cast<size_t>(row) * K;
    float* out_score = a.out_partner_score + static_cast<size_t>(row) * K;
    if (cap4 <= kThreads) {
        // ranks among a warp's 32 candidates first, then among the warps' K best each
        uint32_t* keys = reinterpret_cast<uint32_t*>(queries);                   // 256 words, no longer needed
        uint32_t* kept_keys = reinterpret_cast<uint32_t*>(sel_s + 3 * kDecodeTop);       // nor are the other warps' lists
        int* kept_slots = sel_s + 3 * kDecodeTop + kThreads;
        const int n_kept = ((cap4 + 31) >> 5) * K;
        const uint32_t key = tid < cap4 ? float_key(cand[tid] + 0.0f) : 1u;      // below every score's key, and not 0 (rank_among)
        keys[tid] = key;
        __syncwarp();
        if (32 * warp < cap4) {
            const int rank = rank_among<8>(keys + 32 * warp, 8, key, lane);
            if (rank < K) {
                kept_keys[warp * K + rank] = key;
                kept_slots[warp * K + rank] = tid;
            }
        }
        if (tid < ((n_kept + 3) & ~3) - n_kept) kept_keys[n_kept + tid] = 0u;
        __syncthreads();
        if (tid < n_kept) {
            const int slot = kept_slots[tid], rank = rank_among<4>(kept_keys, (n_kept + 3) >> 2, kept_keys[tid], tid);
            if (rank < K && slot < cap) {
                const float score = cand[slot];
                const int r = bs_shift >= 0 ? (slot - L) >> bs_shift : (slot - L) / bs;
                const int pos = slot < L ? t - L + 1 + slot : sel_s[3 * max(r, 0)] * bs + (slot - L - r * bs);
                out_pos[rank] = score > kNegInf ? pos : t - L + 1;
                out_score[rank] = score;
            }
        }
        // more partners than candidates
        for (int k = cap + tid; k < K; k += kThreads) { out_pos[k] = t - L + 1; out_score[k] = kNegInf; }
    } else if (kCtaTop || cap4 > 512) {
        topk_large(cand, cap, K, L, t, bs, sel_s, out_pos, out_score);
    } else if (warp == 0) {
        topk_warp(cand, cap4, K, L, t, bs, bs_shift, sel, short_list, out_pos, out_score);
    }
}

struct TileArgs {
    SelectArgs base;          // packed mode; queries [n_seq * q_len, ...]; row = b * q_len + t
    int q_len;                // query positions 0 .. q_len - 1 of every sequence
    int tile_queries;         // positions per CTA
    int warp_bytes, stats_bytes, window_rows, param_bytes;
};

template <int kDt, int kTileWarps>
__global__ void __launch_bounds__(32 * kTileWarps, (kDt == RLM_F32 ? 16 : 32) / kTileWarps) relation_select_tile_kernel(const TileArgs m) {
    constexpr bool kFast = kDt != RLM_F32;            // one 16-bit dtype throughout (else run-time dtypes)
    constexpr int kTileThreads = 32 * kTileWarps;
    const int tile_q = m.tile_queries;
    extern __shared__ __align__(128) unsigned char smem[];
    const SelectArgs& a = m.base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int key_dtype = kFast ? kDt : a.key_dtype, stats_dtype = kFast ? kDt : a.stats_dtype,
              query_dtype = kFast ? kDt : a.query_dtype;
    const int tiles_per_seq = (m.q_len + tile_q - 1) / tile_q;
    const int b = blockIdx.x / tiles_per_seq, t0 = (blockIdx.x - b * tiles_per_seq) * tile_q;
    const int t_end = min(t0 + tile_q, m.q_len);               // exclusive
    const int nb = a.n_blocks, bs = a.block_size, L = a.local_window, top = a.top_blocks, K = a.k_out;
    const int bs_shift = (bs & (bs - 1)) == 0 ? 31 - __clz(bs) : -1;
    const int ks = key_dtype == RLM_F32 ? 4 : 2, ss = stats_dtype == RLM_F32 ? 4 : 2;
    const size_t key_row = static_cast<size_t>(kD) * ks, stat_row = static_cast<size_t>(kD) * ss;
    const uint32_t key_stride = static_cast<uint32_t>(key_row), stat_stride = static_cast<uint32_t>(stat_row);
    const int buckets4 = 4 * a.buckets;
    griddep_sync();

    // ---- shared staging: statistics of the blocks complete at the tile's last position, and the
    // union of the local windows: positions [w_lo, t_end)
    // (offsets from `smem`, not a table of pointers indexed at run time: through such a table the compiler loses that
    // they are shared memory, and every load becomes a generic one with a 64-bit address)
    const auto st = [&](int which) { return smem + which * m.stats_bytes; };
    unsigned char* win_a = smem + 4 * m.stats_bytes;
    unsigned char* win_p = win_a + static_cast<size_t>(m.window_rows) * key_stride;
    float* params = reinterpret_cast<float*>(win_p + static_cast<size_t>(m.window_rows) * key_stride);
    unsigned char* warp_base = reinterpret_cast<unsigned char*>(params) + m.param_bytes + static_cast<size_t>(warp) * m.warp_bytes;
    const int n_stage = top > 0 ? min(t_end / bs, nb) : 0;
    const int w_lo = max(t0 - L + 1, 0);
    const size_t seq_stats = static_cast<size_t>(b) * nb * stat_row, seq_keys = static_cast<size_t>(b) * a.max_t * key_row;
    {
        const char* src[4] = {static_cast<const char*>(a.anchor_mean) + seq_stats, static_cast<const char*>(a.anchor_std) + seq_stats,
                              static_cast<const char*>(a.partner_mean) + seq_stats, static_cast<const char*>(a.partner_std) + seq_stats};
        const int stat_cpr = static_cast<int>(stat_row / 16), key_cpr = static_cast<int>(key_row / 16);   // 16-byte chunks per row
        const int stat_chunks = n_stage * stat_cpr;
        for (int i = tid; i < 4 * stat_chunks; i += kTileThreads) {
            const int which = i / stat_chunks, c = i - which * stat_chunks;
            const int r = c / stat_cpr, cc = c - r * stat_cpr;
            cp_async16(smem_u32(st(which)) + r * stat_stride + 16 * cc, src[which] + 16 * c);
        }
        const int win_chunks = (t_end - w_lo) * key_cpr;
        const char* ka = static_cast<const char*>(a.anchor_keys) + seq_keys + w_lo * key_row;
        const char* kp = static_cast<const char*>(a.partner_keys) + seq_keys + w_lo * key_row;
        for (int i = tid; i < win_chunks; i += kTileThreads) {
            const int r = i / key_cpr, cc = i - r * key_cpr;
            cp_async16(smem_u32(win_a) + r * key_stride + 16 * cc, ka + 16 * i);
            cp_async16(smem_u32(win_p) + r * key_stride + 16 * cc, kp + 16 * i);
        }
        cp_async_commit();
    }
    // router parameters, shared by the warps: softplus a[4] p[4], bias a, bias p
    float* sp_a = params, *sp_p = params + 4, *bias_a = params + 8, *bias_p = bias_a + buckets4;
    for (int i = tid; i < buckets4; i += kTileThreads) {
        bias_a[i] = load_scalar(a.anchor_bias, i, a.param_dtype);
        bias_p[i] = load_scalar(a.partner_bias, i, a.param_dtype);
    }
    if (tid < 8) {
        const float gamma = load_scalar(tid < 4 ? a.anchor_gamma : a.partner_gamma, tid & 3, a.param_dtype);
        params[tid] = canon_log(__fadd_rn(1.0f, canon_exp(gamma)));
    }
    // per-warp scratch
    float* queries = reinterpret_cast<float*>(warp_base);                     // aq | arq | pq | prq
    uint32_t* short_list = reinterpret_cast<uint32_t*>(queries + 4 * kD);     // 64 words of the top-K filter
    float* bscore = reinterpret_cast<float*>(short_list + 64);
    float* cand = bscore + ((nb + 3) & ~3);
    const int cap = L + top * bs, cap4 = (cap + 3) & ~3;
    int* sel = reinterpret_cast<int*>(cand + cap4);
    for (int i = cap + lane; i < cap4; i += 32) cand[i] = kNegInf;
    cp_async_wait_all();
    __syncthreads();

    for (int t = t0 + warp; t < t_end; t += kTileWarps) {
        const int row = b * m.q_len + t;
        const int ls = max(t - L + 1, 0), first_local = ls - (t - L + 1);
        const int n_complete = min((t + 1) / bs, nb);
        // this query's rows of the projections
        for (int i = lane; i < 4 * kD; i += 32) {
            float v;
            if (i < kD) v = load_scalar(a.anchor_query, row * a.aq_stride + i, query_dtype);
            else if (i < 2 * kD) v = load_scalar(a.anchor_router_query, row * a.arq_stride + i - kD, query_dtype);
            else v = load_scalar(a.partner_base, row * a.pbase_stride + i - 2 * kD, query_dtype);
            queries[i] = v;
        }
        __syncwarp();
        const float* aq = queries, *arq = queries + kD;
        float* pq = queries + 2 * kD, *prq = queries + 3 * kD;
        // the query's window starts (t - L + 1 - w_lo) rows into the staged union (negative rows are never valid)
        const ptrdiff_t win_off = static_cast<ptrdiff_t>(t - L + 1 - w_lo) * static_cast<ptrdiff_t>(key_stride);
        const unsigned char* local_a = win_a + win_off;
        const unsigned char* local_p = win_p + win_off;
        const unsigned char* seq_a = static_cast<const unsigned char*>(a.anchor_keys) + seq_keys;
        const unsigned char* seq_p = static_cast<const unsigned char*>(a.partner_keys) + seq_keys;
        bool ok = true;
        // ---- anchor
        uint32_t bk = 0;
        int bp = 0x7fffffff;
        if constexpr (kFast) {
            NarrowChunk<kDt> q;
            if (top > 0) {
                load_query_chunk(arq, q);
                score_blocks_warp<kDt>(st(0), st(1), nb, n_complete, bs, t, ls, a.strict_valid, a.buckets, q,
                                  sp_a, bias_a, bscore);
            }
            load_query_chunk(aq, q);
            score_window_warp<kDt>(local_a, L, first_local, t - L + 1, -1, q, nullptr,
                                   0, bk, bp);
            if (top > 0) {
                __syncwarp();
                if (nb <= 128) pick_blocks_warp(bscore, nb, top, bs, ls, sel);
                else pick_blocks(bscore, nb, top, bs, ls, sel);
                score_remote_warp<kDt>(seq_a, top * bs, sel, bs, bs_shift, -1, q, nullptr, 0, bk, bp);
            }
        } else {
            if (top > 0)
                score_blocks_any<kAnyDtype>(st(0), st(1), stats_dtype, nb, n_complete, bs, t, ls, a.strict_valid, a.buckets,
                                        arq, sp_a, bias_a, bscore, 0, 1);
            score_rows_split<kAnyDtype, 1>(local_a, key_dtype, L, nullptr, bs, first_local, t - L + 1, -1, nullptr, 0, aq,
                                       nullptr, 0, 0, 1, bk, bp, 0u, ok);
            if (top > 0) {
                __syncwarp();
                pick_blocks(bscore, nb, top, bs, ls, sel);
                uint32_t rk = 0;
                int rp = 0x7fffffff;
                score_rows_split<kAnyDtype, 1, true>(seq_a, key_dtype, top * bs, sel, bs, 0, 0, -1, nullptr, 0, aq, nullptr, 0,
                                                 0, 1, rk, rp, 0u, ok);
                if (rp != 0x7fffffff && (rk > bk || bp == 0x7fffffff || (rk == bk && rp < bp))) { bk = rk; bp = rp; }
            }
        }
        int anchor_pos = bp;
        if (anchor_pos == 0x7fffffff) { anchor_pos = 0; bk = float_key(kNegInf); }
        if (lane == 0) {
            a.out_anchor[row] = anchor_pos;
            a.out_anchor_score[row] = key_float(bk);
        }
        // ---- partner queries: query-side base + the anchor's cached row
        for (int i = lane; i < 2 * kD; i += 32) {
            const float add = load_scalar(a.partner_anchor_cache,
                                          (static_cast<size_t>(b) * a.max_t + anchor_pos) * 2 * kD + i, key_dtype);
            pq[i] = __fadd_rn(pq[i], add);
        }
        __syncwarp();
        // ---- partners
        uint32_t dk = 0;
        int dp = 0x7fffffff;
        if constexpr (kFast) {
            QueryChunk q;
            if (top > 0) {
                load_query_chunk(prq, q);
                score_blocks_warp<kDt>(st(2), st(3), nb, n_complete, bs, t, ls, a.strict_valid, a.buckets, q,
                                  sp_p, bias_p, bscore);
            }
            load_query_chunk(pq, q);
            score_window_warp<kDt>(local_p, L, first_local, t - L + 1, anchor_pos, q,
                                   cand, 0, dk, dp);
            if (top > 0) {
                __syncwarp();
                if (nb <= 128) pick_blocks_warp(bscore, nb, top, bs, ls, sel);
                else pick_blocks(bscore, nb, top, bs, ls, sel);
                score_remote_warp<kDt>(seq_p, top * bs, sel, bs, bs_shift, anchor_pos, q, cand, L, dk, dp);
            }
        } else {
            if (top > 0)
                score_blocks_any<kAnyDtype>(st(2), st(3), stats_dtype, nb, n_complete, bs, t, ls, a.strict_valid, a.buckets,
                                        prq, sp_p, bias_p, bscore, 0, 1);
            score_rows_split<kAnyDtype, 1>(local_p, key_dtype, L, nullptr, bs, first_local, t - L + 1, anchor_pos, nullptr, 0,
                                       pq, cand, 0, 0, 1, dk, dp, 0u, ok);
            if (top > 0) {
                __syncwarp();
                pick_blocks(bscore, nb, top, bs, ls, sel);
                score_rows_split<kAnyDtype, 1, true>(seq_p, key_dtype, top * bs, sel, bs, 0, 0, anchor_pos, nullptr, 0, pq, cand,
                                                 L, 0, 1, dk, dp, 0u, ok);
            }
        }
        __syncwarp();
        int32_t* out_pos = a.out_partner + static_cast<size_t>(row) * K;
        float* out_sc = a.out_partner_score + static_cast<size_t>(row) * K;
        topk_warp(cand, cap4, K, L, t, bs, bs_shift, sel, short_list, out_pos, out_sc);
        __syncwarp();
    }
}

// ---- whole-sequence multi-anchor selection: the tiled form of relation_select_multi_kernel (one 16-bit dtype)
//
// A CTA of kTileWarps warps serves up to 4 kTileWarps consecutive positions of one sequence; every warp
// keeps its queries and walks them through 2 S phases — the anchors of slot 0 .. S - 1 (each barring
// the positions taken before it), then the partners of slot 0 .. S - 1 (each barring all anchors).
// A phase's block statistics and window union (one slot, one stream) are staged for the whole CTA
// in one of two buffers while the previous phase is being computed.  Rules and arithmetic are
// relation_select_multi_kernel's (same results bit for bit).
struct MultiTileArgs {
    MultiSelectArgs m;
    int q_len, tile_queries;
    int warp_bytes, stats_bytes, param_bytes, stage_bytes;
};

template <int kDt, int kTileWarps>
__global__ void __launch_bounds__(32 * kTileWarps, 32 / kTileWarps) relation_select_multi_tile_kernel(const MultiTileArgs ta) {
    constexpr int kTileThreads = 32 * kTileWarps;
    const int tile_q = ta.tile_queries;
    extern __shared__ __align__(128) unsigned char smem[];
    const MultiSelectArgs& m = ta.m;
    const SelectArgs& a = m.base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = m.slots, K = a.k_out;
    const int tiles_per_seq = (ta.q_len + tile_q - 1) / tile_q;
    const int b = blockIdx.x / tiles_per_seq, t0 = (blockIdx.x - b * tiles_per_seq) * tile_q;
    const int t_end = min(t0 + tile_q, ta.q_len);
    const int nb = a.n_blocks, bs = a.block_size, L = a.local_window, top = a.top_blocks;
    const int bs_shift = (bs & (bs - 1)) == 0 ? 31 - __clz(bs) : -1;
    constexpr size_t key_row = kRow, stat_row = kRow;
    const int buckets4 = 4 * a.buckets;
    griddep_sync();

    // two staging buffers: mean | std | window union of one slot and stream
    const auto stage_buf = [&](int ph) { return smem + (ph & 1) * ta.stage_bytes; };     // an offset, not a table of pointers
    float* params = reinterpret_cast<float*>(smem + 2 * ta.stage_bytes);      // per slot: softplus a[4] p[4], bias a, bias p
    const int slot_params = 8 + 2 * buckets4;
    unsigned char* warp_base = reinterpret_cast<unsigned char*>(params) + ta.param_bytes + static_cast<size_t>(warp) * ta.warp_bytes;
    const int n_stage = top > 0 ? min(t_end / bs, nb) : 0;
    const int w_lo = max(t0 - L + 1, 0);
    auto request_phase = [&](int ph) {
        if (ph < 2 * S) {
            const int s = ph < S ? ph : ph - S;
            const bool partner = ph >= S;
            unsigned char* dst = stage_buf(ph);
            const size_t seq_stats = s * m.stats_slot + static_cast<size_t>(b) * nb * stat_row;
            const size_t seq_keys = s * m.keys_slot + static_cast<size_t>(b) * a.max_t * key_row;
            const char* mean = static_cast<const char*>(partner ? a.partner_mean : a.anchor_mean) + seq_stats;
            const char* stdv = static_cast<const char*>(partner ? a.partner_std : a.anchor_std) + seq_stats;
            const char* keys = static_cast<const char*>(partner ? a.partner_keys : a.anchor_keys) + seq_keys + w_lo * key_row;
            const int stat_chunks = n_stage * 8;
            for (int i = tid; i < 2 * stat_chunks; i += kTileThreads) {
                const int which = i >= stat_chunks, c = i - which * stat_chunks;
                cp_async16(smem_u32(dst) + which * ta.stats_bytes + 16 * c,
                           (which ? stdv : mean) + 16 * c);
            }
            const int win_chunks = (t_end - w_lo) * 8;
            for (int i = tid; i < win_chunks; i += kTileThreads)
                cp_async16(smem_u32(dst) + 2 * ta.stats_bytes + 16 * i, keys + 16 * i);
        }
        cp_async_commit();
    };
    request_phase(0);
    for (int i = tid; i < S * slot_params; i += kTileThreads) {
        const int s = i / slot_params, j = i - s * slot_params;
        float v;
        if (j < 8) {
            const float gamma = load_scalar(slot_ptr(j < 4 ? a.anchor_gamma : a.partner_gamma, s * m.gamma_slot), j & 3, a.param_dtype);
            v = canon_log(__fadd_rn(1.0f, canon_exp(gamma)));
        } else if (j < 8 + buckets4) {
            v = load_scalar(slot_ptr(a.anchor_bias, s * m.bias_slot), j - 8, a.param_dtype);
        } else {
            v = load_scalar(slot_ptr(a.partner_bias, s * m.bias_slot), j - 8 - buckets4, a.param_dtype);
        }
        params[i] = v;
    }
    // per-warp scratch
    float* queries = reinterpret_cast<float*>(warp_base);                     // exact query | router query
    uint32_t* short_list = reinterpret_cast<uint32_t*>(queries + 2 * kD);     // 64 words of the top-K filter
    int* taken = reinterpret_cast<int*>(short_list + 64);                     // [4 queries][kMaxSlots]
    float* bscore = reinterpret_cast<float*>(taken + 4 * kMaxSlots);
    float* cand = bscore + ((nb + 3) & ~3);
    const int cap = L + top * bs, cap4 = (cap + 3) & ~3;
    int* sel = reinterpret_cast<int*>(cand + cap4);
    for (int i = cap + lane; i < cap4; i += 32) cand[i] = kNegInf;
    for (int i = lane; i < 4 * kMaxSlots; i += 32) taken[i] = -1;

    for (int ph = 0; ph < 2 * S; ++ph) {
        request_phase(ph + 1);                       // into the buffer phase ph - 1 has left
        cp_async_wait_group1();
        __syncthreads();                             // phase ph is staged (and, first time, the parameters are written)
        const int s = ph < S ? ph : ph - S;
        const bool partner = ph >= S;
        const unsigned char* st_mean = stage_buf(ph);
        const unsigned char* st_std = st_mean + ta.stats_bytes;
        const unsigned char* win = st_mean + 2 * ta.stats_bytes;
        const float* sp = params + s * slot_params + (partner ? 4 : 0);
        const float* bias = params + s * slot_params + 8 + (partner ? buckets4 : 0);
        const unsigned char* seq_keys = static_cast<const unsigned char*>(partner ? a.partner_keys : a.anchor_keys) +
                                        s * m.keys_slot + static_cast<size_t>(b) * a.max_t * key_row;
        int qi = 0;
        for (int t = t0 + warp; t < t_end; t += kTileWarps, ++qi) {
            const int row = b * ta.q_len + t;
            const int ls = max(t - L + 1, 0), first_local = ls - (t - L + 1);
            const int n_complete = min((t + 1) / bs, nb);
            int* mine = taken + qi * kMaxSlots;
            const unsigned char* local = win + static_cast<ptrdiff_t>(t - L + 1 - w_lo) * static_cast<ptrdiff_t>(kRow);
            ExclRegs ex;
            if (!partner) {
                // ---- anchor of slot s: active iff s <= t; the positions taken by slots 0 .. s - 1 are barred
                int32_t* out_idx = m.out_anchor + static_cast<size_t>(row) * S + s;
                float* out_sc = m.out_anchor_score + static_cast<size_t>(row) * S + s;
                uint8_t* out_live = m.out_anchor_active + static_cast<size_t>(row) * S + s;
                if (s > t) {
                    if (lane == 0) { *out_idx = 0; *out_sc = kNegInf; *out_live = 0; }
                    continue;                        // taken[s] stays -1
                }
                for (int i = lane; i < 2 * kD; i += 32) {
                    const float v = i < kD ? load_scalar(a.anchor_query, row * a.aq_stride + s * kD + i, kDt)
                                           : load_scalar(a.anchor_router_query, row * a.arq_stride + s * kD + i - kD, kDt);
                    queries[i] = v;
                }
                ex.n = s;
#pragma unroll
                for (int x = 0; x < kMaxExclude; ++x) ex.v[x] = x < s ? mine[x] : -1;
                __syncwarp();
                NarrowChunk<kDt> q;
                if (top > 0) {
                    load_query_chunk(queries + kD, q);
                    score_blocks_warp<kDt>(st_mean, st_std, nb, n_complete, bs, t, ls, a.strict_valid, a.buckets, q, sp,
                                      bias, bscore);
                }
                load_query_chunk(queries, q);
                uint32_t bk = 0;
                int bp = 0x7fffffff;
                score_window_warp<kDt, true>(local, L, first_local, t - L + 1, -1, q, nullptr,
                                             0, bk, bp, &ex);
                if (top > 0) {
                    __syncwarp();
                    if (nb <= 128) pick_blocks_warp(bscore, nb, top, bs, ls, sel);
                    else pick_blocks(bscore, nb, top, bs, ls, sel);
                    score_remote_warp<kDt, true>(seq_keys, top * bs, sel, bs, bs_shift, -1, q, nullptr, 0, bk, bp, &ex);
                }
                const float score = bp == 0x7fffffff ? kNegInf : key_float(bk);
                const bool live = score > kNegInf;
                if (lane == 0) {
                    *out_idx = live ? bp : 0;
                    *out_sc = live ? score : kNegInf;
                    *out_live = live ? 1 : 0;
                    mine[s] = live ? bp : -1;
                }
                __syncwarp();
            } else {
                // ---- partners of slot s: none without an anchor; the anchors of all slots are barred
                int32_t* out_idx = m.out_partner + (static_cast<size_t>(row) * S + s) * K;
                float* out_sc = m.out_partner_score + (static_cast<size_t>(row) * S + s) * K;
                const int anchor_pos = mine[s];
                if (anchor_pos < 0) {
                    if (lane < K) { out_idx[lane] = 0; out_sc[lane] = kNegInf; }
                    continue;
                }
                const unsigned char* pac = static_cast<const unsigned char*>(a.partner_anchor_cache) + s * m.pac_slot;
                for (int i = lane; i < 2 * kD; i += 32) {
                    const float base = load_scalar(a.partner_base, row * a.pbase_stride + s * 2 * kD + i, kDt);
                    const float add = load_scalar(pac, (static_cast<size_t>(b) * a.max_t + anchor_pos) * 2 * kD + i, kDt);
                    queries[i] = __fadd_rn(base, add);
                }
                ex.n = S;
#pragma unroll
                for (int x = 0; x < kMaxExclude; ++x) ex.v[x] = x < S ? mine[x] : -1;
                __syncwarp();
                QueryChunk q;
                if (top > 0) {
                    load_query_chunk(queries + kD, q);
                    score_blocks_warp<kDt>(st_mean, st_std, nb, n_complete, bs, t, ls, a.strict_valid, a.buckets, q, sp,
                                      bias, bscore);
                }
                load_query_chunk(queries, q);
                uint32_t dk = 0;
                int dp = 0x7fffffff;
                score_window_warp<kDt, true>(local, L, first_local, t - L + 1, anchor_pos, q,
                                             cand, 0, dk, dp, &ex);
                if (top > 0) {
                    __syncwarp();
                    if (nb <= 128) pick_blocks_warp(bscore, nb, top, bs, ls, sel);
                    else pick_blocks(bscore, nb, top, bs, ls, sel);
                    score_remote_warp<kDt, true>(seq_keys, top * bs, sel, bs, bs_shift, anchor_pos, q, cand, L, dk, dp, &ex);
                }
                __syncwarp();
                bool exact = false;
                if (cap4 <= 128) exact = topk_filter<4>(cand, cap4, K, L, t, bs, bs_shift, sel, short_list, out_idx, out_sc);
                else if (cap4 <= 256) exact = topk_filter<8>(cand, cap4, K, L, t, bs, bs_shift, sel, short_list, out_idx, out_sc);
                else exact = topk_filter<16>(cand, cap4, K, L, t, bs, bs_shift, sel, short_list, out_idx, out_sc);
                if (!exact) {
                    if (cap4 <= 128) topk_tournament<4>(cand, cap4, K, L, t, bs, bs_shift, sel, out_idx, out_sc);
                    else if (cap4 <= 256) topk_tournament<8>(cand, cap4, K, L, t, bs, bs_shift, sel, out_idx, out_sc);
                    else topk_tournament<16>(cand, cap4, K, L, t, bs, bs_shift, sel, out_idx, out_sc);
                    // slots without a finite score report index 0 (written by this very lane just above)
                    if (lane < K && !(out_sc[lane] > kNegInf)) { out_idx[lane] = 0; out_sc[lane] = kNegInf; }
                }
                __syncwarp();
            }
        }
        __syncthreads();                             // everybody has left buffer ph & 1
    }
    cp_async_wait_all();
}

// A tile's shape: warps per CTA and positions per warp.  A launch lasts as many waves of a tile per SM as its tiles
// need, each as long as the tile's rounds of a position per warp; a round of 32 warps fills the SM, fewer warps
// leave issue slots unused but end sooner (relative lengths below from one round of each: 27, 23, 21 and 19 us for
// 512 positions, launch and staging included, and 341, 339, 403 and 477 us for 8 x 4096).  The shape of least waves x
// rounds x length that fits the shared memory is taken: 8 x 4096 positions run as 1024 tiles of 32, 3 x 1984 as 126 of
// 48 (as 249 of 24 they take 53 us, as 186 of 32 67 us), 512 as 64 of 8.  The lengths are those of the single-anchor
// 16-bit builds; the multi-anchor and the fp32 builds follow the same rule without having been measured for it.
struct TileShape { int warps, per_warp, smem_bytes; };

template <typename Smem>
TileShape tile_shape(int n_seq, int q_len, int most_warps, const Smem& smem) {
    static constexpr int kShapes[4][2] = {{32, 32}, {24, 24}, {16, 19}, {8, 13}};
    TileShape best{0, 0, 0};
    int64_t best_cost = INT64_MAX;
    for (const auto& shape : kShapes) {
        const int warps = shape[0];
        if (warps > most_warps || (warps == 24 && most_warps < 32)) continue;
        for (int per_warp = 4; per_warp >= 1; per_warp /= 2) {
            const int total = smem(warps, per_warp * warps);
            if (total > kSmemDynamicLimit) continue;
            const int64_t tiles = static_cast<int64_t>(n_seq) * ((q_len + per_warp * warps - 1) / (per_warp * warps));
            const int64_t waves = (tiles + sm_count() - 1) / sm_count();
            const int64_t cost = waves * (32 * per_warp * shape[1] + shape[1]);      // staging: 1/32 of a round
            if (cost < best_cost) { best_cost = cost; best = {warps, per_warp, total}; }
        }
    }
    return best;
}

// Shared memory a tile asks for.  Tiles of one wave each want an SM of their own, as tile_shape counts on; with 8 or 16
// warps several fit one, and under programmatic launch they crowd on the SMs that the kernel before leaves first.  So
// such a launch asks for more than half of an SM's shared memory (us a pass of a layer: 2 x 848 of d 256, K 4
// 80.6 -> 68.4, 2 x 640 77.3 -> 67.4, 2 x 1024 of d 768 169 -> 159, 1 x 512 52.5 -> 52.5; with the selector alone launched
// in the ordinary way 69.7, 66.1, 160, 52.1; of a multi-anchor stack: 2 x 848 of d 256, two slots 123 -> 101, 1 x 2048 of
// d 512 196 -> 177).  More tiles than SMs share them anyway.
int tile_smem(int total, int tiles, int warps) {
    constexpr int kMoreThanHalf = 228 * 1024 / 2;
    return tiles <= sm_count() && warps <= 16 && total < kMoreThanHalf ? kMoreThanHalf : total;
}

template <int kDt>
auto multi_tile_kernel(int warps) {
    return warps == 32 ? relation_select_multi_tile_kernel<kDt, 32> : warps == 24 ? relation_select_multi_tile_kernel<kDt, 24>
           : warps == 16 ? relation_select_multi_tile_kernel<kDt, 16> : relation_select_multi_tile_kernel<kDt, 8>;
}

template <int kDt>
auto tile_kernel(int warps) {
    return warps == 32 ? relation_select_tile_kernel<kDt, 32> : warps == 24 ? relation_select_tile_kernel<kDt, 24>
           : warps == 16 ? relation_select_tile_kernel<kDt, 16> : relation_select_tile_kernel<kDt, 8>;
}

int launch_multi_tile(MultiTileArgs& ta, void* stream) {
    MultiSelectArgs& m = ta.m;
    SelectArgs& a = m.base;
    if (a.n_seq < 1 || ta.q_len < 1 || ta.q_len > a.max_t || a.max_t < 1 || a.n_blocks < 1 || a.buckets < 1 ||
        a.local_window < 1 || a.top_blocks < 0 || a.max_t % a.n_blocks != 0 || m.slots < 1 || m.slots > kMaxSlots ||
        a.k_out < 1 || a.k_out > kMaxKOut) {
        set_error("relation_select_multi_prefill: sizes must be positive, T a multiple of the block count, 1..8 slots, "
                  "K <= 32, query length <= T");
        return RLM_ERR_SHAPE;
    }
    if ((a.query_dtype != RLM_BF16 && a.query_dtype != RLM_F16) || a.key_dtype != a.query_dtype ||
        a.stats_dtype != a.query_dtype || !valid_dtype(a.param_dtype)) {
        set_error("relation_select_multi_prefill: queries, caches and block statistics must share bfloat16 or float16 "
                  "(relation_select_multi_rows serves the other dtypes)");
        return RLM_ERR_UNSUPPORTED;
    }
    const void* need[] = {a.anchor_query, a.anchor_keys, a.anchor_router_query, a.anchor_mean, a.anchor_std, a.anchor_gamma,
                          a.anchor_bias, a.partner_base, a.partner_anchor_cache, a.partner_keys, a.partner_mean,
                          a.partner_std, a.partner_gamma, a.partner_bias, m.out_anchor, m.out_anchor_score,
                          m.out_anchor_active, m.out_partner, m.out_partner_score};
    for (const void* q : need) if (!q) { set_error("relation_select_multi_prefill: NULL pointer"); return RLM_ERR_NULL; }
    const void* bulk[] = {a.anchor_keys, a.anchor_mean, a.anchor_std, a.partner_keys, a.partner_mean, a.partner_std,
                          a.partner_anchor_cache};
    for (const void* q : bulk)
        if (!aligned16(q)) {
            set_error("relation_select_multi_prefill: key caches, block statistics and the partner-anchor cache must be 16-byte aligned");
            return RLM_ERR_ALIGN;
        }
    a.block_size = a.max_t / a.n_blocks;
    const int cap = a.local_window + a.top_blocks * a.block_size;
    if (cap > 512) {
        set_error("relation_select_multi_prefill: at most 512 candidates per query (window + remote blocks)");
        return RLM_ERR_UNSUPPORTED;
    }
    const int ps = dtype_size(a.param_dtype);
    m.keys_slot = static_cast<size_t>(a.n_seq) * a.max_t * kD * 2;
    m.pac_slot = static_cast<size_t>(a.n_seq) * a.max_t * 2 * kD * 2;
    m.stats_slot = static_cast<size_t>(a.n_seq) * a.n_blocks * kD * 2;
    m.gamma_slot = static_cast<size_t>(4) * ps;
    m.bias_slot = static_cast<size_t>(4) * a.buckets * ps;
    if (a.aq_stride < static_cast<int64_t>(m.slots) * kD || a.arq_stride < static_cast<int64_t>(m.slots) * kD ||
        a.pbase_stride < static_cast<int64_t>(m.slots) * 2 * kD) {
        set_error("relation_select_multi_prefill: a query row stride is shorter than the slots it holds");
        return RLM_ERR_SHAPE;
    }
    const int cap4 = (cap + 3) & ~3;
    const int floats = 2 * kD + 64 + 4 * kMaxSlots + ((a.n_blocks + 3) & ~3) + cap4;
    ta.warp_bytes = align16(floats * 4 + 3 * (a.top_blocks > 0 ? a.top_blocks : 1) * 4) + 16;
    ta.stats_bytes = a.n_blocks * static_cast<int>(kRow);
    ta.param_bytes = align16(m.slots * (8 + 8 * a.buckets) * 4);
    const TileShape shape = tile_shape(a.n_seq, ta.q_len, 32, [&](int warps, int tile) {
        ta.stage_bytes = (2 * ta.stats_bytes + (a.local_window + tile) * static_cast<int>(kRow) + 127) & ~127;
        return 2 * ta.stage_bytes + ta.param_bytes + warps * ta.warp_bytes;
    });
    if (shape.warps == 0) {
        set_error("relation_select_multi_prefill: block statistics + window union exceed 227 KB of shared memory");
        return RLM_ERR_SMEM;
    }
    const int warps = shape.warps, total = shape.smem_bytes;
    ta.tile_queries = shape.per_warp * warps;
    ta.stage_bytes = (2 * ta.stats_bytes + (a.local_window + ta.tile_queries) * static_cast<int>(kRow) + 127) & ~127;
    auto kernel = a.key_dtype == RLM_BF16 ? multi_tile_kernel<RLM_BF16>(warps) : multi_tile_kernel<RLM_F16>(warps);
    int rc = allow_large_smem(reinterpret_cast<const void*>(kernel), kSmemPerCta);
    if (rc != RLM_OK) return rc;
    const int tiles = a.n_seq * ((ta.q_len + ta.tile_queries - 1) / ta.tile_queries);
    launch_kernel(kernel, dim3(tiles), dim3(32 * warps), tile_smem(total, tiles, warps), stream, ta);
    count_launch();
    return check_launch("relation_select_multi_tile_kernel");
}

int tile_warp_bytes(const SelectArgs& a) {
    const int cap4 = (a.local_window + a.top_blocks * a.block_size + 3) & ~3;
    const int floats = 4 * kD + 64 + ((a.n_blocks + 3) & ~3) + cap4;
    return align16(floats * 4 + 3 * (a.top_blocks > 0 ? a.top_blocks : 1) * 4) + 16;
}

int launch_tile(TileArgs& m, void* stream) {
    SelectArgs& a = m.base;
    if (a.n_seq < 1 || m.q_len < 1 || m.q_len > a.max_t || a.max_t < 1 || a.n_blocks < 1 || a.buckets < 1 ||
        a.local_window < 1 || a.top_blocks < 0 || a.max_t % a.n_blocks != 0 || a.k_out < 1 || a.k_out > kMaxKOut) {
        set_error("relation_select_packed_prefill: sizes must be positive, T a multiple of the block count, K <= 32, "
                  "query length <= T");
        return RLM_ERR_SHAPE;
    }
    if (!valid_dtype(a.query_dtype) || !valid_dtype(a.key_dtype) || !valid_dtype(a.stats_dtype) || !valid_dtype(a.param_dtype)) {
        set_error("relation_select_packed_prefill: unknown dtype code");
        return RLM_ERR_DTYPE;
    }
    const void* need[] = {a.anchor_query, a.anchor_keys, a.anchor_router_query, a.anchor_mean, a.anchor_std, a.anchor_gamma,
                          a.anchor_bias, a.partner_base, a.partner_anchor_cache, a.partner_keys, a.partner_mean,
                          a.partner_std, a.partner_gamma, a.partner_bias, a.out_anchor, a.out_anchor_score, a.out_partner,
                          a.out_partner_score};
    for (const void* q : need) if (!q) { set_error("relation_select_packed_prefill: NULL pointer"); return RLM_ERR_NULL; }
    const void* bulk[] = {a.anchor_keys, a.anchor_mean, a.anchor_std, a.partner_keys, a.partner_mean, a.partner_std,
                          a.partner_anchor_cache};
    for (const void* q : bulk)
        if (!aligned16(q)) {
            set_error("relation_select_packed_prefill: key caches, block statistics and the partner-anchor cache must be 16-byte aligned");
            return RLM_ERR_ALIGN;
        }
    a.block_size = a.max_t / a.n_blocks;
    a.mode = kPacked;
    const int cap = a.local_window + a.top_blocks * a.block_size;
    if (cap > 512) {
        set_error("relation_select_packed_prefill: at most 512 candidates per query (window + remote blocks)");
        return RLM_ERR_UNSUPPORTED;
    }
    const bool fast = a.query_dtype != RLM_F32 && a.key_dtype == a.query_dtype && a.stats_dtype == a.query_dtype;
    const int key_stride = kD * dtype_size(a.key_dtype), stat_stride = kD * dtype_size(a.stats_dtype);
    m.warp_bytes = tile_warp_bytes(a);
    m.stats_bytes = align16(a.n_blocks * stat_stride);
    m.param_bytes = align16((8 + 8 * a.buckets) * 4);
    const TileShape shape = tile_shape(a.n_seq, m.q_len, fast ? 32 : 16, [&](int warps, int tile) {
        return 4 * m.stats_bytes + 2 * (a.local_window + tile) * key_stride + m.param_bytes + warps * m.warp_bytes;
    });
    if (shape.warps == 0) {
        set_error("relation_select_packed_prefill: block statistics + window union exceed 227 KB of shared memory");
        return RLM_ERR_SMEM;
    }
    const int warps = shape.warps, total = shape.smem_bytes;
    m.tile_queries = shape.per_warp * warps;
    m.window_rows = a.local_window + m.tile_queries;
    auto kernel = !fast ? (warps == 16 ? relation_select_tile_kernel<RLM_F32, 16> : relation_select_tile_kernel<RLM_F32, 8>)
                  : a.key_dtype == RLM_BF16 ? tile_kernel<RLM_BF16>(warps) : tile_kernel<RLM_F16>(warps);
    int rc = allow_large_smem(reinterpret_cast<const void*>(kernel), kSmemPerCta);
    if (rc != RLM_OK) return rc;
    const int tiles = a.n_seq * ((m.q_len + m.tile_queries - 1) / m.tile_queries);
    launch_kernel(kernel, dim3(tiles), dim3(32 * warps), tile_smem(total, tiles, warps), stream, m);
    count_launch();
    return check_launch("relation_select_tile_kernel");
}

// The decode form in one dtype has the kernel of warp passes; launches of more rows than the SMs hold at once
// (rows in flight count there, not a row's chain) and the other forms take a select_row build.
template <int kDt>
auto select_kernel(bool many_rows, bool decode, bool passes, bool resident) {
    return resident ? relation_select_decode_kernel<kDt, true>
           : passes && !many_rows ? relation_select_decode_kernel<kDt, false>
           : many_rows ? (decode ? relation_select_kernel<4, kDt, true> : relation_select_kernel<4, kDt, false>)
                       : relation_select_kernel<3, kDt, false>;
}

auto select_kernel_fp32(bool many_rows, bool decode, bool passes, bool resident, bool cta_top) {
    return resident ? (cta_top ? relation_select_decode_kernel<RLM_F32, true, true> : relation_select_decode_kernel<RLM_F32, true>)
           : passes && !many_rows ? (cta_top ? relation_select_decode_kernel<RLM_F32, false, true> : relation_select_decode_kernel<RLM_F32, false>)
           : decode ? (many_rows ? relation_select_kernel<4, RLM_F32, true> : relation_select_kernel<3, RLM_F32, true>)
                    : (many_rows ? relation_select_kernel<4, kAnyDtype, false> : relation_select_kernel<3, kAnyDtype, false>);
}

int launch(SelectArgs& a, void* stream) {
    if (a.n_rows == 0) return RLM_OK;
    bool many_rows = false;
    const int ready = prepare(a, many_rows, true);
    if (ready != RLM_OK) return ready;
    const Plan& plan = a.plan;
    const int dtype = a.key_dtype == a.query_dtype && a.stats_dtype == a.query_dtype ? a.query_dtype : kAnyDtype;
    const bool decode = a.mode == kPacked && !a.row_batch && !a.row_position && !a.exclude_list;
    // Single precision: two such CTAs per SM, three of the general form, which therefore holds more rows at once; and the
    // many rounds of choosing short blocks are no shorter here (us with whole caches not staged, general form -> this one:
    // 512 positions in blocks of 8, top 8 11.3 -> 11.6, top 4 10.4 -> 10.3).
    const bool passes = decode && a.top_blocks <= kDecodeTop && plan.total <= kSmemDynamicLimit - kDecodeStatic &&
                        (dtype != RLM_F32 || (a.n_rows <= 2 * a.sm_count && (a.resident || a.block_size >= 16 || a.top_blocks <= 4)));
    // Picked rows are read where they lie: with a buffer for them only one CTA of a wide choice fitted an SM (us, 149 rows of
    // 352 positions in fp32, eight blocks of 32: 19.0 -> 11.3, 15.1 in the general form).
    if (passes && !many_rows && !a.resident)
        a.plan = make_plan(a.n_blocks, a.block_size, a.local_window, a.top_blocks, a.buckets, dtype_size(a.key_dtype),
                           dtype_size(a.stats_dtype), a.mode, false, 0, false);
    auto kernel = dtype == RLM_BF16 ? select_kernel<RLM_BF16>(many_rows, decode, passes, a.resident)
                  : dtype == RLM_F16 ? select_kernel<RLM_F16>(many_rows, decode, passes, a.resident)
                  : dtype == RLM_F32 ? select_kernel_fp32(many_rows, decode, passes, a.resident, a.local_window + a.top_blocks * a.block_size > 256)
                                     : (many_rows ? relation_select_kernel<4, kAnyDtype, false> : relation_select_kernel<3, kAnyDtype, false>);
    int rc = allow_large_smem(reinterpret_cast<const void*>(kernel), kSmemPerCta);
    if (rc != RLM_OK) return rc;
    launch_kernel(kernel, dim3(a.n_rows), dim3(kThreads), plan.total, stream, a);
    count_launch();
    return check_launch("relation_select_kernel");
}

int launch_multi(MultiSelectArgs& m, void* stream) {
    SelectArgs& a = m.base;
    if (a.n_rows == 0) return RLM_OK;
    if (a.n_rows < 0 || a.n_seq < 1 || a.max_t < 1 || a.n_blocks < 1 || a.buckets < 1 || a.local_window < 1 ||
        a.top_blocks < 0 || a.max_t % a.n_blocks != 0 || m.slots < 1 || m.slots > kMaxSlots || a.k_out < 1 ||
        a.k_out > kMaxKOut) {
        set_error("relation_select_multi_rows: sizes must be positive, T a multiple of the block count, 1..8 slots, K <= 32");
        return RLM_ERR_SHAPE;
    }
    if (!valid_dtype(a.query_dtype) || !valid_dtype(a.key_dtype) || !valid_dtype(a.stats_dtype) || !valid_dtype(a.param_dtype)) {
        set_error("relation_select_multi_rows: unknown dtype code");
        return RLM_ERR_DTYPE;
    }
    const void* need[] = {a.anchor_query, a.anchor_keys, a.anchor_router_query, a.anchor_mean, a.anchor_std, a.anchor_gamma,
                          a.anchor_bias, a.partner_base, a.partner_anchor_cache, a.partner_keys, a.partner_mean,
                          a.partner_std, a.partner_gamma, a.partner_bias, a.row_batch, a.row_position, m.out_anchor,
                          m.out_anchor_score, m.out_anchor_active, m.out_partner, m.out_partner_score};
    for (const void* q : need) if (!q) { set_error("relation_select_multi_rows: NULL pointer"); return RLM_ERR_NULL; }
    const void* bulk[] = {a.anchor_keys, a.anchor_mean, a.anchor_std, a.partner_keys, a.partner_mean, a.partner_std,
                          a.partner_anchor_cache};
    for (const void* q : bulk)
        if (!aligned16(q)) {
            set_error("relation_select_multi_rows: key caches, block statistics and the partner-anchor cache must be 16-byte aligned");
            return RLM_ERR_ALIGN;
        }
    a.block_size = a.max_t / a.n_blocks;
    a.shared_streams = 0;
    a.sm_count = sm_count();
    const int ks = dtype_size(a.key_dtype), ss = dtype_size(a.stats_dtype), ps = dtype_size(a.param_dtype);
    m.plan_anchor = make_plan(a.n_blocks, a.block_size, a.local_window, a.top_blocks, a.buckets, ks, ss, kAnchorOnly, false);
    m.plan_partner = make_plan(a.n_blocks, a.block_size, a.local_window, a.top_blocks, a.buckets, ks, ss, kPartnerOnly, false);
    const int total = m.plan_anchor.total > m.plan_partner.total ? m.plan_anchor.total : m.plan_partner.total;
    if (total > kSmemDynamicLimit) {
        set_error("relation_select_multi_rows: block statistics + local window + remote blocks exceed 227 KB of shared memory");
        return RLM_ERR_SMEM;
    }
    m.keys_slot = static_cast<size_t>(a.n_seq) * a.max_t * kD * ks;
    m.pac_slot = static_cast<size_t>(a.n_seq) * a.max_t * 2 * kD * ks;
    m.stats_slot = static_cast<size_t>(a.n_seq) * a.n_blocks * kD * ss;
    m.gamma_slot = static_cast<size_t>(4) * ps;
    m.bias_slot = static_cast<size_t>(4) * a.buckets * ps;
    if (a.aq_stride < static_cast<int64_t>(m.slots) * kD || a.arq_stride < static_cast<int64_t>(m.slots) * kD ||
        a.pbase_stride < static_cast<int64_t>(m.slots) * 2 * kD) {
        set_error("relation_select_multi_rows: a query row stride is shorter than the slots it holds");
        return RLM_ERR_SHAPE;
    }
    const int dtype = a.key_dtype == a.query_dtype && a.stats_dtype == a.query_dtype ? a.query_dtype : kAnyDtype;
    auto kernel = dtype == RLM_BF16 ? relation_select_multi_kernel<RLM_BF16>
                  : dtype == RLM_F16 ? relation_select_multi_kernel<RLM_F16> : relation_select_multi_kernel<kAnyDtype>;
    int rc = allow_large_smem(reinterpret_cast<const void*>(kernel), kSmemPerCta);
    if (rc != RLM_OK) return rc;
    launch_kernel(kernel, dim3(a.n_rows), dim3(kThreads), total, stream, m);
    count_launch();
    return check_launch("relation_select_multi_kernel");
}

}  // namespace
}  // namespace rlm

extern "C" int rlm_relation_select_packed_prefill(
    const void* anchor_query, const void* anchor_keys, const void* anchor_router_query,
    const void* anchor_mean, const void* anchor_std, const void* anchor_gamma, const void* anchor_bias,
    const void* partner_base, const void* partner_anchor_cache, const void* partner_keys,
    const void* partner_mean, const void* partner_std, const void* partner_gamma, const void* partner_bias,
    int32_t* out_anchor, float* out_anchor_score, int32_t* out_partner, float* out_partner_score,
    int64_t anchor_query_stride, int64_t anchor_router_query_stride, int64_t partner_base_stride,
    int n_seq, int query_length, int max_t, int n_blocks, int buckets, int local_window, int top_blocks, int k_out,
    int strict_valid, int query_dtype, int key_dtype, int stats_dtype, int param_dtype, int32_t* status,
    void* stream) {
    rlm::TileArgs m{};
    rlm::SelectArgs& a = m.base;
    a.aq_stride = anchor_query_stride; a.arq_stride = anchor_router_query_stride; a.pbase_stride = partner_base_stride;
    a.anchor_query = anchor_query; a.anchor_keys = anchor_keys; a.anchor_router_query = anchor_router_query;
    a.anchor_mean = anchor_mean; a.anchor_std = anchor_std; a.anchor_gamma = anchor_gamma; a.anchor_bias = anchor_bias;
    a.partner_base = partner_base; a.partner_anchor_cache = partner_anchor_cache; a.partner_keys = partner_keys;
    a.partner_mean = partner_mean; a.partner_std = partner_std; a.partner_gamma = partner_gamma; a.partner_bias = partner_bias;
    a.out_anchor = out_anchor; a.out_anchor_score = out_anchor_score; a.out_partner = out_partner;
    a.out_partner_score = out_partner_score; a.status = status;
    a.n_rows = n_seq * query_length; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks; a.buckets = buckets;
    a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = k_out; a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    m.q_len = query_length;
    return rlm::launch_tile(m, stream);
}

extern "C" int rlm_relation_select_multi_prefill(
    const void* anchor_query, const void* anchor_keys, const void* anchor_router_query,
    const void* anchor_mean, const void* anchor_std, const void* anchor_gamma, const void* anchor_bias,
    const void* partner_base, const void* partner_anchor_cache, const void* partner_keys,
    const void* partner_mean, const void* partner_std, const void* partner_gamma, const void* partner_bias,
    int32_t* out_anchor, float* out_anchor_score, uint8_t* out_anchor_active, int32_t* out_partner,
    float* out_partner_score, int64_t anchor_query_stride, int64_t anchor_router_query_stride,
    int64_t partner_base_stride, int query_length, int n_seq, int slots, int max_t, int n_blocks, int buckets,
    int local_window, int top_blocks, int k_out, int strict_valid, int query_dtype, int key_dtype, int stats_dtype,
    int param_dtype, int32_t* status, void* stream) {
    if (n_seq == 0 || query_length == 0) return RLM_OK;
    rlm::MultiTileArgs ta{};
    rlm::MultiSelectArgs& m = ta.m;
    rlm::SelectArgs& a = m.base;
    a.anchor_query = anchor_query; a.anchor_keys = anchor_keys; a.anchor_router_query = anchor_router_query;
    a.anchor_mean = anchor_mean; a.anchor_std = anchor_std; a.anchor_gamma = anchor_gamma; a.anchor_bias = anchor_bias;
    a.partner_base = partner_base; a.partner_anchor_cache = partner_anchor_cache; a.partner_keys = partner_keys;
    a.partner_mean = partner_mean; a.partner_std = partner_std; a.partner_gamma = partner_gamma; a.partner_bias = partner_bias;
    a.status = status; a.n_rows = n_seq * query_length; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks;
    a.buckets = buckets; a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = k_out;
    a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    a.aq_stride = anchor_query_stride; a.arq_stride = anchor_router_query_stride; a.pbase_stride = partner_base_stride;
    m.slots = slots; m.out_anchor = out_anchor; m.out_anchor_score = out_anchor_score;
    m.out_anchor_active = out_anchor_active; m.out_partner = out_partner; m.out_partner_score = out_partner_score;
    ta.q_len = query_length;
    return rlm::launch_multi_tile(ta, stream);
}

extern "C" int rlm_relation_select_multi_rows(
    const void* anchor_query, const void* anchor_keys, const void* anchor_router_query,
    const void* anchor_mean, const void* anchor_std, const void* anchor_gamma, const void* anchor_bias,
    const void* partner_base, const void* partner_anchor_cache, const void* partner_keys,
    const void* partner_mean, const void* partner_std, const void* partner_gamma, const void* partner_bias,
    const int32_t* row_batch, const int32_t* row_position, int32_t* out_anchor, float* out_anchor_score,
    uint8_t* out_anchor_active, int32_t* out_partner, float* out_partner_score,
    int64_t anchor_query_stride, int64_t anchor_router_query_stride, int64_t partner_base_stride,
    int n_rows, int n_seq, int slots,
    int max_t, int n_blocks, int buckets, int local_window, int top_blocks, int k_out, int strict_valid,
    int query_dtype, int key_dtype, int stats_dtype, int param_dtype, int32_t* status, void* stream) {
    rlm::MultiSelectArgs m{};
    rlm::SelectArgs& a = m.base;
    a.anchor_query = anchor_query; a.anchor_keys = anchor_keys; a.anchor_router_query = anchor_router_query;
    a.anchor_mean = anchor_mean; a.anchor_std = anchor_std; a.anchor_gamma = anchor_gamma; a.anchor_bias = anchor_bias;
    a.partner_base = partner_base; a.partner_anchor_cache = partner_anchor_cache; a.partner_keys = partner_keys;
    a.partner_mean = partner_mean; a.partner_std = partner_std; a.partner_gamma = partner_gamma; a.partner_bias = partner_bias;
    a.row_batch = row_batch; a.row_position = row_position; a.status = status;
    a.n_rows = n_rows; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks; a.buckets = buckets;
    a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = k_out; a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    a.aq_stride = anchor_query_stride; a.arq_stride = anchor_router_query_stride; a.pbase_stride = partner_base_stride;
    m.slots = slots; m.out_anchor = out_anchor; m.out_anchor_score = out_anchor_score;
    m.out_anchor_active = out_anchor_active; m.out_partner = out_partner; m.out_partner_score = out_partner_score;
    return rlm::launch_multi(m, stream);
}

extern "C" int rlm_relation_select_packed(
    const void* anchor_query, const void* anchor_keys, const void* anchor_router_query,
    const void* anchor_mean, const void* anchor_std, const void* anchor_gamma,
    const void* anchor_bias, const void* partner_base, const void* partner_anchor_cache,
    const void* partner_keys, const void* partner_mean, const void* partner_std,
    const void* partner_gamma, const void* partner_bias, const int64_t* position,
    const int32_t* row_batch, const int32_t* row_position, int32_t* out_anchor,
    float* out_anchor_score, int32_t* out_partner, float* out_partner_score,
    int64_t anchor_query_stride, int64_t anchor_router_query_stride, int64_t partner_base_stride,
    int n_rows, int n_seq,
    int max_t, int n_blocks, int buckets, int local_window, int top_blocks, int k_out,
    int strict_valid, int query_dtype, int key_dtype, int stats_dtype, int param_dtype,
    int32_t* status, void* stream) {
    rlm::SelectArgs a{};
    a.aq_stride = anchor_query_stride; a.arq_stride = anchor_router_query_stride; a.pbase_stride = partner_base_stride;
    a.anchor_query = anchor_query; a.anchor_keys = anchor_keys; a.anchor_router_query = anchor_router_query;
    a.anchor_mean = anchor_mean; a.anchor_std = anchor_std; a.anchor_gamma = anchor_gamma; a.anchor_bias = anchor_bias;
    a.partner_base = partner_base; a.partner_anchor_cache = partner_anchor_cache; a.partner_keys = partner_keys;
    a.partner_mean = partner_mean; a.partner_std = partner_std; a.partner_gamma = partner_gamma; a.partner_bias = partner_bias;
    a.position = position; a.row_batch = row_batch; a.row_position = row_position;
    a.out_anchor = out_anchor; a.out_anchor_score = out_anchor_score; a.out_partner = out_partner; a.out_partner_score = out_partner_score;
    a.status = status;
    a.n_rows = n_rows; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks; a.buckets = buckets;
    a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = k_out; a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    a.mode = rlm::kPacked;
    return rlm::launch(a, stream);
}

extern "C" int rlm_anchor_select(
    const void* anchor_query, const void* anchor_keys, const void* router_query,
    const void* block_mean, const void* block_std, const void* gamma, const void* bias,
    const int64_t* position, const int32_t* row_batch, const int32_t* row_position,
    const int32_t* exclude_index, int exclude_count,
    int32_t* out_index, float* out_score, int n_rows, int n_seq, int max_t, int n_blocks,
    int buckets, int local_window, int top_blocks, int strict_valid, int query_dtype,
    int key_dtype, int stats_dtype, int param_dtype, int32_t* status, void* stream) {
    rlm::SelectArgs a{};
    a.exclude_list = exclude_index; a.exclude_count = exclude_count;
    a.aq_stride = 64; a.arq_stride = 64;
    a.anchor_query = anchor_query; a.anchor_keys = anchor_keys; a.anchor_router_query = router_query;
    a.anchor_mean = block_mean; a.anchor_std = block_std; a.anchor_gamma = gamma; a.anchor_bias = bias;
    a.position = position; a.row_batch = row_batch; a.row_position = row_position;
    a.out_anchor = out_index; a.out_anchor_score = out_score; a.status = status;
    a.n_rows = n_rows; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks; a.buckets = buckets;
    a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = 0; a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    a.mode = rlm::kAnchorOnly;
    return rlm::launch(a, stream);
}

extern "C" int rlm_partner_topk(
    const void* partner_query, const void* partner_keys, const void* router_query,
    const void* block_mean, const void* block_std, const void* gamma, const void* bias,
    const int64_t* position, const int32_t* row_batch, const int32_t* row_position,
    const int32_t* anchor_index, const int32_t* exclude_index, int exclude_count,
    int32_t* out_index, float* out_score, int n_rows, int n_seq,
    int max_t, int n_blocks, int buckets, int local_window, int top_blocks, int k_out,
    int strict_valid, int query_dtype, int key_dtype, int stats_dtype, int param_dtype,
    int32_t* status, void* stream) {
    rlm::SelectArgs a{};
    a.exclude_list = exclude_index; a.exclude_count = exclude_count;
    a.pbase_stride = 64; a.prq_stride = 64;
    a.partner_base = partner_query; a.partner_router_query = router_query; a.partner_keys = partner_keys;
    a.partner_mean = block_mean; a.partner_std = block_std; a.partner_gamma = gamma; a.partner_bias = bias;
    a.position = position; a.row_batch = row_batch; a.row_position = row_position;
    a.anchor_index_in = anchor_index; a.out_partner = out_index; a.out_partner_score = out_score; a.status = status;
    a.n_rows = n_rows; a.n_seq = n_seq; a.max_t = max_t; a.n_blocks = n_blocks; a.buckets = buckets;
    a.local_window = local_window; a.top_blocks = top_blocks; a.k_out = k_out; a.strict_valid = strict_valid != 0;
    a.query_dtype = query_dtype; a.key_dtype = key_dtype; a.stats_dtype = stats_dtype; a.param_dtype = param_dtype;
    a.mode = rlm::kPartnerOnly;
    return rlm::launch(a, stream);
}


// torch.library operators of the package, registered from native code: argument checks, output
// allocation and the C-ABI call without a Python frame in between.
//
// What bounds an operator of a decode position is the host: its kernel takes 3-15 us, the same
// operator written as a Python custom operator 30-40 us of interpreter time (schema binding, autograd
// and mutation wrappers, ~40 boxed ctypes arguments).  Registered here a call costs the dispatcher and
// the launch.  Names, schemas and error types are those of the Python definitions they stand in for:
// operators the reference project defines (src/relation_lm/kernels/relation_select.py:311,
// triton_select.py:255-298, router_cache.py:175, relation_reduce.py:149-420) and this library's
// extensions.  Fake implementations and documentation stay in the Python modules.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/record_function.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <initializer_list>
#include <mutex>
#include <optional>
#include <tuple>
#include <vector>

#include "../../include/relation_lm_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using Two = std::tuple<Tensor, Tensor>;
using Four = std::tuple<Tensor, Tensor, Tensor, Tensor>;
using Five = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>;
using Six = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor>;

// ------------------------------------------------------------------ checks

struct Named {
    const char* name;
    const Tensor* t;      // nullptr: an optional argument that is absent
};
#define ARG(x) Named{#x, &(x)}
#define OPT(x) Named{#x, (x).has_value() ? &*(x) : nullptr}

void require_cuda(const Named& a) {
    TORCH_CHECK_NOT_IMPLEMENTED(a.t->is_cuda(), a.name, " is on ", a.t->device(),
                                ": relation_lm operators run on CUDA devices only");
}

c10::Device contiguous(std::initializer_list<Named> args) {
    const Tensor* first = nullptr;
    for (const Named& a : args) {
        if (!a.t) continue;
        require_cuda(a);
        if (!first) first = a.t;
        TORCH_CHECK_VALUE(a.t->device() == first->device(), a.name, " is on ", a.t->device(), ", expected ", first->device());
        TORCH_CHECK_VALUE(a.t->is_contiguous(), a.name, " must be contiguous");
    }
    return first->device();
}

// 2-D tensors whose rows are dense (unit inner stride); the row stride is free.
c10::Device dense_rows(std::initializer_list<Named> args) {
    const Tensor* first = args.begin()->t;
    for (const Named& a : args) {
        require_cuda(a);
        TORCH_CHECK_VALUE(a.t->dim() == 2 && a.t->stride(1) == 1, a.name, " must be 2-D with unit inner stride");
        TORCH_CHECK_VALUE(a.t->device() == first->device(), a.name, " is on ", a.t->device(), ", expected ", first->device());
    }
    return first->device();
}

void require_position(const Tensor& position, c10::Device device) {
    TORCH_CHECK_VALUE(position.device() == device && position.scalar_type() == at::kLong && position.numel() == 1,
                      "position must be a one-element int64 tensor on the operands' device");
}

int code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return RLM_F32;
        case at::kBFloat16: return RLM_BF16;
        case at::kHalf: return RLM_F16;
        default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t.scalar_type(), "; use float32, bfloat16 or float16");
    }
    return -1;
}

int same_dtype(const char* what, std::initializer_list<const Tensor*> ts) {
    const Tensor* first = *ts.begin();
    for (const Tensor* t : ts)
        TORCH_CHECK_VALUE(t->scalar_type() == first->scalar_type(), what, " tensors must share one dtype, got ",
                          first->scalar_type(), " and ", t->scalar_type());
    return code(*first);
}

bool is_shape(const Tensor& t, at::IntArrayRef shape) { return t.sizes() == shape; }
bool is_f32(const Tensor& t) { return t.scalar_type() == at::kFloat; }
bool is_i32(const Tensor& t) { return t.scalar_type() == at::kInt; }

// ------------------------------------------------------------------ launch context

// The per-device word kernels OR their error bits into.  Allocated at a device's first launch and kept
// for the life of the process (never destroyed: the CUDA context may be gone before static destructors).
Tensor& status_word(int index) {
    static std::mutex mutex;
    static Tensor* words = new Tensor[64];
    TORCH_CHECK(index >= 0 && index < 64, "unexpected CUDA device index");
    std::lock_guard<std::mutex> lock(mutex);
    if (!words[index].defined())
        words[index] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, static_cast<c10::DeviceIndex>(index)));
    return words[index];
}

struct Launch {
    c10::cuda::CUDAGuard guard;
    void* stream;
    int32_t* status;
    explicit Launch(c10::Device device)
        : guard(device), stream(c10::cuda::getCurrentCUDAStream(device.index()).stream()),
          status(status_word(device.index()).data_ptr<int32_t>()) {}
};

void check(int rc) {
    if (rc == RLM_OK) return;
    const char* text = rlm_last_error();
    const std::string message = text && *text ? text : "status " + std::to_string(rc);
    if (rc == RLM_ERR_LAUNCH) TORCH_CHECK(false, message);
    TORCH_CHECK_VALUE(false, message);
}

Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, c10::Device device) {
    return Tensor(at::detail::empty_cuda(shape, dtype, device, std::nullopt));
}

void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
float* f32(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
float* f32(const OptTensor& t) { return t.has_value() ? f32(*t) : nullptr; }
int32_t* i32(const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); }
int64_t* i64(const Tensor& t) { return static_cast<int64_t*>(t.data_ptr()); }

// ------------------------------------------------------------------ selection

struct SelectTensors {
    const Tensor &anchor_query, &anchor_keys, &anchor_router_query, &anchor_block_mean, &anchor_block_std, &anchor_gamma,
        &anchor_bias, &partner_base, &partner_anchor_cache, &partner_keys, &partner_block_mean, &partner_block_std,
        &partner_gamma, &partner_bias;

    c10::Device caches() const {
        return contiguous({ARG(anchor_keys), ARG(anchor_block_mean), ARG(anchor_block_std), ARG(anchor_gamma),
                           ARG(anchor_bias), ARG(partner_anchor_cache), ARG(partner_keys), ARG(partner_block_mean),
                           ARG(partner_block_std), ARG(partner_gamma), ARG(partner_bias)});
    }
    void rows() const { dense_rows({ARG(anchor_query), ARG(anchor_router_query), ARG(partner_base)}); }
    int query_dtype() const { return same_dtype("query", {&anchor_query, &anchor_router_query, &partner_base}); }
    int key_dtype() const { return same_dtype("key cache", {&anchor_keys, &partner_keys, &partner_anchor_cache}); }
    int stats_dtype() const {
        return same_dtype("block statistics", {&anchor_block_mean, &anchor_block_std, &partner_block_mean, &partner_block_std});
    }
    int param_dtype() const { return same_dtype("gamma/bias", {&anchor_gamma, &anchor_bias, &partner_gamma, &partner_bias}); }
};

#define SELECT_PARAMS                                                                                                    \
    const Tensor &anchor_query, const Tensor &anchor_keys, const Tensor &anchor_router_query,                            \
        const Tensor &anchor_block_mean, const Tensor &anchor_block_std, const Tensor &anchor_gamma,                     \
        const Tensor &anchor_bias, const Tensor &partner_base, const Tensor &partner_anchor_cache,                       \
        const Tensor &partner_keys, const Tensor &partner_block_mean, const Tensor &partner_block_std,                   \
        const Tensor &partner_gamma, const Tensor &partner_bias
#define SELECT_TENSORS                                                                                                   \
    SelectTensors {                                                                                                      \
        anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std, anchor_gamma, anchor_bias,  \
            partner_base, partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std, partner_gamma,      \
            partner_bias                                                                                                 \
    }
#define SELECT_POINTERS(s)                                                                                               \
    ptr((s).anchor_query), ptr((s).anchor_keys), ptr((s).anchor_router_query), ptr((s).anchor_block_mean),               \
        ptr((s).anchor_block_std), ptr((s).anchor_gamma), ptr((s).anchor_bias), ptr((s).partner_base),                   \
        ptr((s).partner_anchor_cache), ptr((s).partner_keys), ptr((s).partner_block_mean), ptr((s).partner_block_std),   \
        ptr((s).partner_gamma), ptr((s).partner_bias)

void check_router_width(const Tensor& query, const Tensor& block_mean) {
    TORCH_CHECK_VALUE(query.size(1) == 64 && block_mean.dim() >= 4 && block_mean.size(2) * block_mean.size(3) == 64 &&
                          block_mean.size(3) == 16,
                      "this build supports gate width 64 with 4 router heads of width 16");
}

Four select(const SelectTensors& s, const Tensor* position, const Tensor* row_batch, const Tensor* row_position,
            int64_t local_window, int64_t top_blocks, int64_t k_out, bool strict_valid) {
    s.rows();
    const c10::Device device = s.caches();
    if (row_batch) {
        const c10::Device rows_device = contiguous({Named{"row_batch", row_batch}, Named{"row_position", row_position}});
        TORCH_CHECK_VALUE(rows_device == device, "row_batch is on ", rows_device, ", expected ", device);
    }
    const int64_t rows = s.anchor_query.size(0);
    check_router_width(s.anchor_query, s.anchor_block_mean);
    TORCH_CHECK_VALUE(s.partner_base.size(1) == 128, "this build supports gate width 64 with 4 router heads of width 16");
    if (position) require_position(*position, device);
    const int q = s.query_dtype(), k = s.key_dtype(), st = s.stats_dtype(), p = s.param_dtype();
    Launch launch(device);
    Tensor anchor = empty({rows}, at::kInt, device), anchor_score = empty({rows}, at::kFloat, device);
    Tensor partner = empty({rows, k_out}, at::kInt, device), partner_score = empty({rows, k_out}, at::kFloat, device);
    check(rlm_relation_select_packed(
        SELECT_POINTERS(s), position ? i64(*position) : nullptr, row_batch ? i32(*row_batch) : nullptr,
        row_position ? i32(*row_position) : nullptr, i32(anchor), f32(anchor_score), i32(partner), f32(partner_score),
        s.anchor_query.stride(0), s.anchor_router_query.stride(0), s.partner_base.stride(0), rows, s.anchor_keys.size(0),
        s.anchor_keys.size(1), s.anchor_block_mean.size(1), s.anchor_bias.size(1), local_window, top_blocks, k_out,
        strict_valid, q, k, st, p, launch.status, launch.stream));
    return {anchor, anchor_score, partner, partner_score};
}

Four relation_select_packed(SELECT_PARAMS, const Tensor& position, int64_t local_window, int64_t top_blocks, int64_t k_out,
                            bool strict_valid) {
    return select(SELECT_TENSORS, &position, nullptr, nullptr, local_window, top_blocks, k_out, strict_valid);
}

Four relation_select_packed_rows(SELECT_PARAMS, const Tensor& row_batch, const Tensor& row_position, int64_t local_window,
                                 int64_t top_blocks, int64_t k_out, bool strict_valid) {
    TORCH_CHECK_VALUE(is_i32(row_batch) && is_i32(row_position), "row_batch and row_position must be int32");
    TORCH_CHECK_VALUE(row_batch.numel() == anchor_query.size(0) && row_position.numel() == anchor_query.size(0),
                      "row_batch and row_position need one entry per query row");
    return select(SELECT_TENSORS, nullptr, &row_batch, &row_position, local_window, top_blocks, k_out, strict_valid);
}

// `fits`: where to say that the tile's staging exceeds the shared memory (nothing was launched), instead of raising.
Four select_prefill(const SelectTensors& s, int64_t query_length, int64_t local_window, int64_t top_blocks, int64_t k_out,
                    bool strict_valid, bool* fits) {
    s.rows();
    const c10::Device device = s.caches();
    const int64_t n_seq = s.anchor_keys.size(0), rows = n_seq * query_length;
    TORCH_CHECK_VALUE(is_shape(s.anchor_query, {rows, 64}) && is_shape(s.anchor_router_query, {rows, 64}) &&
                          is_shape(s.partner_base, {rows, 128}),
                      "queries must hold one row per (sequence, position): [B * query_length, width]");
    check_router_width(s.anchor_query, s.anchor_block_mean);
    const int q = s.query_dtype(), k = s.key_dtype(), st = s.stats_dtype(), p = s.param_dtype();
    Launch launch(device);
    Tensor anchor = empty({rows}, at::kInt, device), anchor_score = empty({rows}, at::kFloat, device);
    Tensor partner = empty({rows, k_out}, at::kInt, device), partner_score = empty({rows, k_out}, at::kFloat, device);
    const int rc = rlm_relation_select_packed_prefill(
        SELECT_POINTERS(s), i32(anchor), f32(anchor_score), i32(partner), f32(partner_score), s.anchor_query.stride(0),
        s.anchor_router_query.stride(0), s.partner_base.stride(0), n_seq, query_length, s.anchor_keys.size(1),
        s.anchor_block_mean.size(1), s.anchor_bias.size(1), local_window, top_blocks, k_out, strict_valid, q, k, st, p,
        launch.status, launch.stream);
    if (fits) *fits = rc != RLM_ERR_SMEM;
    if (!fits || *fits) check(rc);
    return {anchor, anchor_score, partner, partner_score};
}

Four relation_select_packed_prefill(SELECT_PARAMS, int64_t query_length, int64_t local_window, int64_t top_blocks,
                                    int64_t k_out, bool strict_valid) {
    return select_prefill(SELECT_TENSORS, query_length, local_window, top_blocks, k_out, strict_valid, nullptr);
}

// Shared by the two multi-anchor forms: shapes, outputs and the call.  The kernels write the anchors'
// activity as bytes 0 / 1, which is the storage of a bool tensor.
Five select_multi(const char* name, const SelectTensors& s, const Tensor* row_batch, const Tensor* row_position,
                 int64_t query_length, int64_t local_window, int64_t top_blocks, int64_t k_out, bool strict_valid) {
    for (const Named& a : {Named{"anchor_query", &s.anchor_query}, Named{"anchor_router_query", &s.anchor_router_query},
                           Named{"partner_base", &s.partner_base}})
        TORCH_CHECK_VALUE(a.t->is_cuda() && a.t->dim() == 3 && a.t->stride(2) == 1 && a.t->stride(1) == a.t->size(2), a.name,
                          " must be a CUDA tensor [N, S, width] whose slots are contiguous inside a row "
                          "(the row stride is free: a column slice of one projection is fine)");
    const c10::Device device = s.caches();
    TORCH_CHECK_VALUE(s.anchor_query.size(2) == 64, "anchor_query must be [N, S, 64]");
    const int64_t rows = s.anchor_query.size(0), slots = s.anchor_query.size(1);
    TORCH_CHECK_VALUE(slots <= 8, "at most 8 anchor slots");
    TORCH_CHECK_VALUE(s.anchor_keys.dim() == 4 && s.anchor_keys.size(0) == slots && s.anchor_keys.size(3) == 64,
                      "anchor_keys must be [S, B, T, 64]");
    const int64_t batch = s.anchor_keys.size(1), max_t = s.anchor_keys.size(2), nb = s.anchor_block_mean.size(2);
    if (!row_batch)
        TORCH_CHECK_VALUE(rows == batch * query_length && query_length >= 1 && query_length <= max_t,
                          "the queries must be the positions 0 .. query_length - 1 of every sequence");
    TORCH_CHECK_VALUE(is_shape(s.anchor_router_query, {rows, slots, 64}) && is_shape(s.partner_base, {rows, slots, 128}) &&
                          is_shape(s.partner_anchor_cache, {slots, batch, max_t, 128}) &&
                          s.partner_keys.sizes() == s.anchor_keys.sizes() &&
                          is_shape(s.anchor_block_mean, {slots, batch, nb, 4, 16}) &&
                          s.partner_block_mean.sizes() == s.anchor_block_mean.sizes() && is_shape(s.anchor_gamma, {slots, 4}) &&
                          s.anchor_bias.dim() == 3 && s.anchor_bias.size(0) == slots && s.anchor_bias.size(1) == 4,
                      name, ": inconsistent shapes");
    if (row_batch) {
        contiguous({Named{"row_batch", row_batch}, Named{"row_position", row_position}});
        TORCH_CHECK_VALUE(is_i32(*row_batch) && is_i32(*row_position) && row_batch->numel() == rows &&
                              row_position->numel() == rows && row_batch->device() == device,
                          "row_batch and row_position must be int32 with one entry per query row");
    }
    const int q = s.query_dtype(), k = s.key_dtype(), st = s.stats_dtype(), p = s.param_dtype();
    Launch launch(device);
    Tensor anchor = empty({rows, slots}, at::kInt, device), anchor_score = empty({rows, slots}, at::kFloat, device);
    Tensor active = empty({rows, slots}, at::kBool, device);
    Tensor partner = empty({rows, slots, k_out}, at::kInt, device), score = empty({rows, slots, k_out}, at::kFloat, device);
    uint8_t* active_bytes = static_cast<uint8_t*>(active.data_ptr());
    if (row_batch)
        check(rlm_relation_select_multi_rows(
            SELECT_POINTERS(s), i32(*row_batch), i32(*row_position), i32(anchor), f32(anchor_score), active_bytes, i32(partner),
            f32(score), s.anchor_query.stride(0), s.anchor_router_query.stride(0), s.partner_base.stride(0), rows, batch, slots,
            max_t, nb, s.anchor_bias.size(2), local_window, top_blocks, k_out, strict_valid, q, k, st, p, launch.status,
            launch.stream));
    else
        check(rlm_relation_select_multi_prefill(
            SELECT_POINTERS(s), i32(anchor), f32(anchor_score), active_bytes, i32(partner), f32(score),
            s.anchor_query.stride(0), s.anchor_router_query.stride(0), s.partner_base.stride(0), query_length, batch, slots,
            max_t, nb, s.anchor_bias.size(2), local_window, top_blocks, k_out, strict_valid, q, k, st, p, launch.status,
            launch.stream));
    return {anchor, anchor_score, active, partner, score};
}

Six with_partner_active(const Five& s) {
    return std::tuple_cat(s, std::make_tuple(at::isfinite(std::get<4>(s))));
}

Six relation_select_multi_rows(SELECT_PARAMS, const Tensor& row_batch, const Tensor& row_position, int64_t local_window,
                               int64_t top_blocks, int64_t partners_per_anchor, bool strict_valid) {
    return with_partner_active(select_multi("relation_select_multi_rows", SELECT_TENSORS, &row_batch, &row_position, 0,
                                            local_window, top_blocks, partners_per_anchor, strict_valid));
}

Six relation_select_multi_prefill(SELECT_PARAMS, int64_t query_length, int64_t local_window, int64_t top_blocks,
                                  int64_t partners_per_anchor, bool strict_valid) {
    return with_partner_active(select_multi("relation_select_multi_prefill", SELECT_TENSORS, nullptr, nullptr, query_length,
                                            local_window, top_blocks, partners_per_anchor, strict_valid));
}

// ... without the partners' activity (finite scores), four elementwise launches that the fused layer has no use for
Five relation_select_multi_prefill_scores(SELECT_PARAMS, int64_t query_length, int64_t local_window, int64_t top_blocks,
                                          int64_t partners_per_anchor, bool strict_valid) {
    return select_multi("relation_select_multi_prefill", SELECT_TENSORS, nullptr, nullptr, query_length, local_window,
                        top_blocks, partners_per_anchor, strict_valid);
}

Two anchor_select(const Tensor& anchor_query, const Tensor& anchor_keys, const Tensor& router_query, const Tensor& block_mean,
                  const Tensor& block_std, const Tensor& gamma, const Tensor& bias, const Tensor& position,
                  int64_t local_window, int64_t top_blocks, bool strict_valid) {
    const c10::Device device = contiguous({ARG(anchor_query), ARG(anchor_keys), ARG(router_query), ARG(block_mean),
                                           ARG(block_std), ARG(gamma), ARG(bias)});
    check_router_width(anchor_query, block_mean);
    require_position(position, device);
    const int64_t rows = anchor_query.size(0);
    const int q = same_dtype("query", {&anchor_query, &router_query}), k = code(anchor_keys);
    const int st = same_dtype("block statistics", {&block_mean, &block_std}), p = same_dtype("gamma/bias", {&gamma, &bias});
    Launch launch(device);
    Tensor index = empty({rows}, at::kInt, device), score = empty({rows}, at::kFloat, device);
    check(rlm_anchor_select(ptr(anchor_query), ptr(anchor_keys), ptr(router_query), ptr(block_mean), ptr(block_std), ptr(gamma),
                            ptr(bias), i64(position), nullptr, nullptr, nullptr, 0, i32(index), f32(score), rows,
                            anchor_keys.size(0), anchor_keys.size(1), block_mean.size(1), bias.size(1), local_window,
                            top_blocks, strict_valid, q, k, st, p, launch.status, launch.stream));
    return {index, score};
}

Two partner_topk(const Tensor& partner_query, const Tensor& partner_keys, const Tensor& router_query, const Tensor& block_mean,
                 const Tensor& block_std, const Tensor& gamma, const Tensor& bias, const Tensor& position,
                 const Tensor& anchor_index, int64_t local_window, int64_t top_blocks, int64_t k_out, bool strict_valid) {
    const c10::Device device = contiguous({ARG(partner_query), ARG(partner_keys), ARG(router_query), ARG(block_mean),
                                           ARG(block_std), ARG(gamma), ARG(bias), ARG(anchor_index)});
    check_router_width(partner_query, block_mean);
    require_position(position, device);
    TORCH_CHECK_VALUE(is_i32(anchor_index), "anchor_index must be int32");
    const int64_t rows = partner_query.size(0);
    const int q = same_dtype("query", {&partner_query, &router_query}), k = code(partner_keys);
    const int st = same_dtype("block statistics", {&block_mean, &block_std}), p = same_dtype("gamma/bias", {&gamma, &bias});
    Launch launch(device);
    Tensor index = empty({rows, k_out}, at::kInt, device), score = empty({rows, k_out}, at::kFloat, device);
    check(rlm_partner_topk(ptr(partner_query), ptr(partner_keys), ptr(router_query), ptr(block_mean), ptr(block_std),
                           ptr(gamma), ptr(bias), i64(position), nullptr, nullptr, i32(anchor_index), nullptr, 0, i32(index),
                           f32(score), rows, partner_keys.size(0), partner_keys.size(1), block_mean.size(1), bias.size(1),
                           local_window, top_blocks, k_out, strict_valid, q, k, st, p, launch.status, launch.stream));
    return {index, score};
}

// ------------------------------------------------------------------ router state

#define ROUTER_PARAMS                                                                                                    \
    Tensor &anchor_raw_cache, Tensor &partner_raw_cache, Tensor &anchor_conv_cache, Tensor &partner_conv_cache,          \
        Tensor &anchor_mean, Tensor &anchor_std, Tensor &partner_mean, Tensor &partner_std,                              \
        const Tensor &anchor_conv_weight, const Tensor &partner_conv_weight
#define ROUTER_ARGS                                                                                                      \
    ARG(anchor_raw_cache), ARG(partner_raw_cache), ARG(anchor_conv_cache), ARG(partner_conv_cache), ARG(anchor_mean),    \
        ARG(anchor_std), ARG(partner_mean), ARG(partner_std), ARG(anchor_conv_weight), ARG(partner_conv_weight)
#define ROUTER_VALUES                                                                                                    \
    anchor_raw_cache, partner_raw_cache, anchor_conv_cache, partner_conv_cache, anchor_mean, anchor_std, partner_mean,   \
        partner_std, anchor_conv_weight, partner_conv_weight
#define ROUTER_POINTERS                                                                                                  \
    ptr(anchor_raw_cache), ptr(partner_raw_cache), ptr(anchor_conv_cache), ptr(partner_conv_cache), ptr(anchor_mean),    \
        ptr(anchor_std), ptr(partner_mean), ptr(partner_std), ptr(anchor_conv_weight), ptr(partner_conv_weight)
#define ROUTER_DTYPES                                                                                                    \
    same_dtype("router cache", {&anchor_raw_cache, &partner_raw_cache, &anchor_conv_cache, &partner_conv_cache}),        \
        same_dtype("block statistics", {&anchor_mean, &anchor_std, &partner_mean, &partner_std}),                        \
        same_dtype("conv weight", {&anchor_conv_weight, &partner_conv_weight})

Tensor router_cache_update(const Tensor& anchor_raw, const Tensor& partner_raw, ROUTER_PARAMS, const Tensor& position,
                           int64_t block_size) {
    const c10::Device device = contiguous({ROUTER_ARGS});
    for (const Named& a : {ARG(anchor_raw), ARG(partner_raw)})
        TORCH_CHECK_VALUE(a.t->device() == device && a.t->dim() == 2 && a.t->size(1) == 64 && a.t->stride(1) == 1, a.name,
                          " must be a [B, 64] CUDA tensor with unit inner stride");
    require_position(position, device);
    const int64_t batch = anchor_raw.size(0);
    // a block's statistics are 64 values, split into heads or not
    TORCH_CHECK_VALUE(anchor_raw_cache.size(2) == 64 && anchor_mean.dim() >= 3 &&
                          c10::multiply_integers(anchor_mean.sizes().slice(2)) == 64,
                      "this build supports router width 64");
    Launch launch(device);
    Tensor out = empty({batch, 2, 64}, at::kFloat, device);
    check(rlm_router_cache_update(ptr(anchor_raw), anchor_raw.stride(0), ptr(partner_raw), partner_raw.stride(0),
                                  ROUTER_POINTERS, i64(position), f32(out), batch, anchor_raw_cache.size(1),
                                  anchor_mean.size(1), block_size, same_dtype("raw key", {&anchor_raw, &partner_raw}),
                                  ROUTER_DTYPES, launch.status, launch.stream));
    return out;
}

void sparse_cache_append(const Tensor& packed, Tensor& anchor_keys, Tensor& partner_keys, Tensor& operand_cache,
                         Tensor& partner_anchor_cache, ROUTER_PARAMS, const Tensor& position, int64_t block_size) {
    const c10::Device device = contiguous({ARG(anchor_keys), ARG(partner_keys), ARG(operand_cache), ARG(partner_anchor_cache),
                                           ROUTER_ARGS});
    dense_rows({ARG(packed)});
    require_position(position, device);
    TORCH_CHECK_VALUE(operand_cache.dim() == 4, "caches must be [layers, B, T, width] and packed [B, layers * (384 + R)]");
    const int64_t layers = operand_cache.size(0), batch = operand_cache.size(1), max_t = operand_cache.size(2),
                  rdim = operand_cache.size(3);
    TORCH_CHECK_VALUE(is_shape(packed, {batch, layers * (384 + rdim)}) && is_shape(anchor_keys, {layers, batch, max_t, 64}) &&
                          is_shape(partner_anchor_cache, {layers, batch, max_t, 128}) &&
                          is_shape(anchor_raw_cache, {layers, batch, max_t, 64}) && anchor_mean.size(0) == layers,
                      "caches must be [layers, B, T, width] and packed [B, layers * (384 + R)]");
    same_dtype("cache", {&anchor_keys, &partner_keys, &operand_cache, &partner_anchor_cache, &anchor_raw_cache});
    Launch launch(device);
    check(rlm_sparse_cache_append(ptr(packed), packed.stride(0), rdim, ptr(anchor_keys), ptr(partner_keys), ptr(operand_cache),
                                  ptr(partner_anchor_cache), ROUTER_POINTERS, i64(position), nullptr, layers, batch, max_t,
                                  anchor_mean.size(2), block_size, code(packed), ROUTER_DTYPES, launch.status, launch.stream));
}

void router_cache_prefill(const Tensor& anchor_raw, const Tensor& partner_raw, ROUTER_PARAMS, int64_t block_size) {
    const c10::Device device = contiguous({ROUTER_ARGS});
    for (const Named& a : {ARG(anchor_raw), ARG(partner_raw)})
        TORCH_CHECK_VALUE(a.t->device() == device && a.t->dim() == 3 && a.t->size(2) == 64 && a.t->stride(2) == 1, a.name,
                          " must be a [B, length, 64] CUDA tensor with unit inner stride");
    TORCH_CHECK_VALUE(partner_raw.sizes() == anchor_raw.sizes(), "anchor_raw and partner_raw must have the same shape");
    Launch launch(device);
    check(rlm_router_cache_prefill(ptr(anchor_raw), anchor_raw.stride(1), anchor_raw.stride(0), ptr(partner_raw),
                                   partner_raw.stride(1), partner_raw.stride(0), ROUTER_POINTERS, anchor_raw.size(1),
                                   anchor_raw.size(0), anchor_raw_cache.size(1), anchor_mean.size(1), block_size,
                                   same_dtype("raw key", {&anchor_raw, &partner_raw}), ROUTER_DTYPES, launch.stream));
}

std::vector<Tensor> sequence_state(const Tensor& packed, int64_t slots, int64_t relation_dim, int64_t block_size,
                                   const Tensor& anchor_conv_weight, const Tensor& partner_conv_weight) {
    const c10::Device device = contiguous({ARG(packed), ARG(anchor_conv_weight), ARG(partner_conv_weight)});
    const int64_t n = slots > 0 ? slots : 1;
    TORCH_CHECK_VALUE(packed.dim() == 3 && slots >= 0 && block_size >= 1 && packed.size(2) == 384 * n + relation_dim &&
                          anchor_conv_weight.numel() == n * 192 && partner_conv_weight.numel() == n * 192,
                      "packed must be [B, T, 384 * slots + R] and the conv weights [slots, 64, 3]");
    const int64_t batch = packed.size(0), length = packed.size(1);
    const int dtype = code(packed), weight = same_dtype("conv weight", {&anchor_conv_weight, &partner_conv_weight});
    Launch launch(device);
    const auto make = [&](std::initializer_list<int64_t> tail, bool slotted) {
        std::vector<int64_t> shape;
        if (slotted && slots > 0) shape.push_back(slots);
        shape.push_back(batch);
        shape.insert(shape.end(), tail);
        return empty(shape, packed.scalar_type(), device);
    };
    const int64_t nb = length / block_size;
    std::vector<Tensor> t = {make({length, 64}, true), make({length, 64}, true), make({length, relation_dim}, false),
                             make({length, 128}, true)};
    for (int i = 0; i < 4; ++i) t.push_back(make({length, 64}, true));
    for (int i = 0; i < 4; ++i) t.push_back(make({nb, 4, 16}, true));
    check(rlm_sequence_state(ptr(packed), packed.size(2), slots, relation_dim, ptr(t[0]), ptr(t[1]), ptr(t[2]), ptr(t[3]),
                             ptr(t[4]), ptr(t[5]), ptr(t[6]), ptr(t[7]), ptr(t[8]), ptr(t[9]), ptr(t[10]), ptr(t[11]),
                             ptr(anchor_conv_weight), ptr(partner_conv_weight), batch, length, block_size, dtype, weight,
                             launch.stream));
    return t;
}

// ------------------------------------------------------------------ relation hidden rows

void check_indices(const Tensor& anchor_index, const Tensor& partner_index, int64_t rows) {
    TORCH_CHECK_VALUE(is_i32(anchor_index) && is_i32(partner_index), "anchor_index and partner_index must be int32");
    TORCH_CHECK_VALUE(anchor_index.numel() == rows && partner_index.dim() == 2 && partner_index.size(0) == rows,
                      "anchor_index must be [B] and partner_index [B, K]");
}

// `out` absent: a new fp32 tensor.  `row_batch` absent: row i reads sequence i.
Tensor hidden_cached(const Tensor* out, const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                     const Tensor& partner_index, const Tensor& product_weight, const Tensor* row_batch) {
    const c10::Device device = contiguous({Named{"out", out}, ARG(expanded_cache), ARG(operand_cache), ARG(anchor_index),
                                           ARG(partner_index), ARG(product_weight), Named{"row_batch", row_batch}});
    TORCH_CHECK_VALUE(operand_cache.dim() == 3 && product_weight.dim() == 2 && partner_index.dim() == 2,
                      "expected operand_cache [B, T, R], product_weight [H, R] and partner_index [N, K]");
    const int64_t n_seq = operand_cache.size(0), max_t = operand_cache.size(1), rdim = operand_cache.size(2);
    const int64_t rows = row_batch ? partner_index.size(0) : n_seq, k_out = partner_index.size(1), hdim = product_weight.size(0);
    check_indices(anchor_index, partner_index, rows);
    if (row_batch)
        TORCH_CHECK_VALUE(is_i32(*row_batch) && row_batch->numel() == rows,
                          "row_batch must be int32 with one entry per query row");
    TORCH_CHECK_VALUE(is_shape(expanded_cache, {n_seq, max_t, 2 * hdim}) && product_weight.size(1) == rdim,
                      "expanded_cache must be [B, T, 2H] and product_weight [H, R]");
    if (out) TORCH_CHECK_VALUE(is_shape(*out, {rows, k_out, hdim}), "out must be [N, K, H]");
    const int cache_dtype = same_dtype("cache", {&expanded_cache, &operand_cache});
    Launch launch(device);
    Tensor result = out ? *out : empty({rows, k_out, hdim}, at::kFloat, device);
    check(rlm_relation_hidden_cached(ptr(expanded_cache), ptr(operand_cache), i32(anchor_index), i32(partner_index),
                                     ptr(product_weight), row_batch ? i32(*row_batch) : nullptr, ptr(result), rows, n_seq,
                                     max_t, rdim, hdim, k_out, cache_dtype, code(product_weight), code(result),
                                     launch.status, launch.stream));
    return result;
}

Tensor relation_hidden_cached(const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                              const Tensor& partner_index, const Tensor& product_weight) {
    return hidden_cached(nullptr, expanded_cache, operand_cache, anchor_index, partner_index, product_weight, nullptr);
}
void relation_hidden_cached_out(Tensor& out, const Tensor& expanded_cache, const Tensor& operand_cache,
                                const Tensor& anchor_index, const Tensor& partner_index, const Tensor& product_weight) {
    hidden_cached(&out, expanded_cache, operand_cache, anchor_index, partner_index, product_weight, nullptr);
}
Tensor relation_hidden_cached_rows(const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                                   const Tensor& partner_index, const Tensor& product_weight, const Tensor& row_batch) {
    return hidden_cached(nullptr, expanded_cache, operand_cache, anchor_index, partner_index, product_weight, &row_batch);
}
void relation_hidden_cached_rows_out(Tensor& out, const Tensor& expanded_cache, const Tensor& operand_cache,
                                     const Tensor& anchor_index, const Tensor& partner_index, const Tensor& product_weight,
                                     const Tensor& row_batch) {
    hidden_cached(&out, expanded_cache, operand_cache, anchor_index, partner_index, product_weight, &row_batch);
}

Tensor hidden_cache_update(const Tensor* out, Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                           const Tensor& partner_index, const Tensor& anchor_weight, const Tensor& partner_weight,
                           const Tensor& product_weight, const Tensor& first_bias, const Tensor& position) {
    const c10::Device device = contiguous({Named{"out", out}, ARG(expanded_cache), ARG(operand_cache), ARG(anchor_index),
                                           ARG(partner_index), ARG(anchor_weight), ARG(partner_weight), ARG(product_weight),
                                           ARG(first_bias)});
    require_position(position, device);
    TORCH_CHECK_VALUE(operand_cache.dim() == 3 && product_weight.dim() == 2 && partner_index.dim() == 2,
                      "expected operand_cache [B, T, R], weights [H, R] and partner_index [B, K]");
    const int64_t batch = operand_cache.size(0), max_t = operand_cache.size(1), rdim = operand_cache.size(2);
    const int64_t hdim = product_weight.size(0), k_out = partner_index.size(1);
    check_indices(anchor_index, partner_index, batch);
    TORCH_CHECK_VALUE(is_shape(expanded_cache, {batch, max_t, 2 * hdim}) && product_weight.size(1) == rdim &&
                          anchor_weight.sizes() == product_weight.sizes() && partner_weight.sizes() == product_weight.sizes() &&
                          first_bias.numel() == hdim,
                      "expected expanded_cache [B, T, 2H], weights [H, R] and first_bias [H]");
    if (out) TORCH_CHECK_VALUE(is_shape(*out, {batch, k_out, hdim}), "expected out [B, K, H] and expanded_cache [B, T, 2H]");
    const int cache_dtype = same_dtype("cache", {&expanded_cache, &operand_cache});
    const int weight_dtype = same_dtype("weight", {&anchor_weight, &partner_weight, &product_weight, &first_bias});
    Launch launch(device);
    Tensor result = out ? *out : empty({batch, k_out, hdim}, at::kFloat, device);
    check(rlm_relation_hidden_cache_update(ptr(expanded_cache), ptr(operand_cache), i32(anchor_index), i32(partner_index),
                                           ptr(anchor_weight), ptr(partner_weight), ptr(product_weight), ptr(first_bias),
                                           i64(position), ptr(result), batch, max_t, rdim, hdim, k_out, cache_dtype,
                                           weight_dtype, code(result), launch.status, launch.stream));
    return result;
}

Tensor relation_hidden_cache_update(Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                                    const Tensor& partner_index, const Tensor& anchor_weight, const Tensor& partner_weight,
                                    const Tensor& product_weight, const Tensor& first_bias, const Tensor& position) {
    return hidden_cache_update(nullptr, expanded_cache, operand_cache, anchor_index, partner_index, anchor_weight,
                               partner_weight, product_weight, first_bias, position);
}
void relation_hidden_cache_update_out(Tensor& out, Tensor& expanded_cache, const Tensor& operand_cache,
                                      const Tensor& anchor_index, const Tensor& partner_index, const Tensor& anchor_weight,
                                      const Tensor& partner_weight, const Tensor& product_weight, const Tensor& first_bias,
                                      const Tensor& position) {
    hidden_cache_update(&out, expanded_cache, operand_cache, anchor_index, partner_index, anchor_weight, partner_weight,
                        product_weight, first_bias, position);
}

void expanded_cache_append(Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_weight,
                           const Tensor& partner_weight, const Tensor& first_bias, const Tensor& position) {
    const c10::Device device = contiguous({ARG(expanded_cache), ARG(operand_cache), ARG(anchor_weight), ARG(partner_weight),
                                           ARG(first_bias)});
    require_position(position, device);
    TORCH_CHECK_VALUE(operand_cache.dim() == 4 && expanded_cache.dim() == 4 && anchor_weight.dim() == 3,
                      "expected stacked tensors: caches [L, B, T, .], weights [L, H, R], bias [L, H]");
    const int64_t layers = operand_cache.size(0), batch = operand_cache.size(1), max_t = operand_cache.size(2),
                  rdim = operand_cache.size(3), hdim = anchor_weight.size(1);
    TORCH_CHECK_VALUE(is_shape(expanded_cache, {layers, batch, max_t, 2 * hdim}) &&
                          is_shape(anchor_weight, {layers, hdim, rdim}) && partner_weight.sizes() == anchor_weight.sizes() &&
                          is_shape(first_bias, {layers, hdim}),
                      "expected expanded_cache [L, B, T, 2H], weights [L, H, R] and first_bias [L, H]");
    const int dtype = same_dtype("caches, weights and bias: 16-bit",
                                 {&expanded_cache, &operand_cache, &anchor_weight, &partner_weight, &first_bias});
    Launch launch(device);
    check(rlm_expanded_cache_append(ptr(expanded_cache), ptr(operand_cache), ptr(anchor_weight), ptr(partner_weight),
                                    ptr(first_bias), i64(position), layers, batch, max_t, rdim, hdim, dtype, launch.status,
                                    launch.stream));
}

void expanded_cache_append_packed(Tensor& expanded_cache, const Tensor& packed, const Tensor& anchor_weight,
                                  const Tensor& partner_weight, const Tensor& first_bias, const Tensor& position) {
    const c10::Device device = contiguous({ARG(expanded_cache), ARG(anchor_weight), ARG(partner_weight), ARG(first_bias)});
    dense_rows({ARG(packed)});
    require_position(position, device);
    TORCH_CHECK_VALUE(expanded_cache.dim() == 4 && anchor_weight.dim() == 3,
                      "expected expanded_cache [L, B, T, 2H], packed [B, L * (384 + R)], weights [L, H, R]");
    const int64_t layers = expanded_cache.size(0), batch = expanded_cache.size(1), max_t = expanded_cache.size(2);
    const int64_t hdim = anchor_weight.size(1), rdim = anchor_weight.size(2);
    TORCH_CHECK_VALUE(expanded_cache.size(3) == 2 * hdim && is_shape(anchor_weight, {layers, hdim, rdim}) &&
                          partner_weight.sizes() == anchor_weight.sizes() && is_shape(first_bias, {layers, hdim}) &&
                          is_shape(packed, {batch, layers * (384 + rdim)}),
                      "expected expanded_cache [L, B, T, 2H], packed [B, L * (384 + R)], weights [L, H, R], bias [L, H]");
    const int dtype = same_dtype("cache, packed rows, weights and bias: 16-bit",
                                 {&expanded_cache, &anchor_weight, &partner_weight, &first_bias, &packed});
    Launch launch(device);
    check(rlm_expanded_cache_append_packed(ptr(expanded_cache), ptr(packed), packed.stride(0), 384 + rdim, 128,
                                           ptr(anchor_weight), ptr(partner_weight), ptr(first_bias), i64(position), layers,
                                           batch, max_t, rdim, hdim, dtype, launch.status, launch.stream));
}

// ------------------------------------------------------------------ norm and reduction

struct ReduceShape { int64_t rows, k_out, dim; };

ReduceShape reduce_shape(const Tensor& raw, const Tensor& partner_scores) {
    TORCH_CHECK_VALUE(raw.dim() == 3 && is_shape(partner_scores, {raw.size(0), raw.size(1)}) && is_f32(partner_scores),
                      "partner_scores must be float32 [B, K]");
    return {raw.size(0), raw.size(1), raw.size(2)};
}

void check_residual(const ReduceShape& s, const Tensor& hidden, const Tensor& mix) {
    TORCH_CHECK_VALUE(is_shape(hidden, {s.rows, s.dim}) && is_f32(hidden) && is_f32(mix) && mix.numel() == 1,
                      "hidden must be float32 [B, D] and mix a one-element float32 tensor");
}

void check_next_norm(const ReduceShape& s, const Tensor& normalized, const Tensor& weight, const Tensor& bias) {
    TORCH_CHECK_VALUE(is_shape(normalized, {s.rows, s.dim}) && is_f32(weight) && is_f32(bias) && weight.numel() == s.dim,
                      "normalized must be [B, D] and the next LayerNorm parameters float32 [D]");
}

Tensor norm_reduce(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight, const Tensor& norm_bias,
                   const Tensor* position, const Tensor* row_position, double norm_eps) {
    const c10::Device device = contiguous({ARG(raw), ARG(partner_scores), ARG(norm_weight), ARG(norm_bias),
                                           Named{"row_position", row_position}});
    if (position) require_position(*position, device);
    const ReduceShape s = reduce_shape(raw, partner_scores);
    if (row_position)
        TORCH_CHECK_VALUE(is_i32(*row_position) && row_position->numel() == s.rows,
                          "row_position must be int32 with one entry per row");
    const int param = same_dtype("norm parameter", {&norm_weight, &norm_bias});
    Launch launch(device);
    Tensor out = empty({s.rows, s.dim}, at::kFloat, device);
    check(rlm_relation_norm_reduce(ptr(raw), f32(partner_scores), ptr(norm_weight), ptr(norm_bias),
                                   position ? i64(*position) : nullptr, row_position ? i32(*row_position) : nullptr,
                                   static_cast<float>(norm_eps), f32(out), nullptr, nullptr, nullptr, nullptr, 0.0f, nullptr, 0,
                                   1, 0, nullptr, s.rows, s.k_out, s.dim, code(raw), param, launch.status, launch.stream));
    return out;
}

Tensor relation_norm_reduce(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight, const Tensor& norm_bias,
                            const Tensor& position, double norm_eps) {
    return norm_reduce(raw, partner_scores, norm_weight, norm_bias, &position, nullptr, norm_eps);
}
Tensor relation_norm_reduce_rows(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight,
                                 const Tensor& norm_bias, const Tensor& row_position, double norm_eps) {
    return norm_reduce(raw, partner_scores, norm_weight, norm_bias, nullptr, &row_position, norm_eps);
}

void relation_norm_reduce_residual(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight,
                                   const Tensor& norm_bias, const Tensor& position, double norm_eps, Tensor& hidden,
                                   const Tensor& mix) {
    const c10::Device device = contiguous({ARG(raw), ARG(partner_scores), ARG(norm_weight), ARG(norm_bias), ARG(hidden),
                                           ARG(mix)});
    require_position(position, device);
    const ReduceShape s = reduce_shape(raw, partner_scores);
    check_residual(s, hidden, mix);
    const int param = same_dtype("norm parameter", {&norm_weight, &norm_bias});
    Launch launch(device);
    check(rlm_relation_norm_reduce(ptr(raw), f32(partner_scores), ptr(norm_weight), ptr(norm_bias), i64(position), nullptr,
                                   static_cast<float>(norm_eps), nullptr, f32(hidden), f32(mix), nullptr, nullptr, 0.0f,
                                   nullptr, 0, 1, 0, nullptr, s.rows, s.k_out, s.dim, code(raw), param, launch.status,
                                   launch.stream));
}

void relation_norm_reduce_residual_norm(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight,
                                        const Tensor& norm_bias, const Tensor& position, double norm_eps, Tensor& hidden,
                                        const Tensor& mix, const Tensor& next_norm_weight, const Tensor& next_norm_bias,
                                        double next_norm_eps, Tensor& normalized) {
    const c10::Device device = contiguous({ARG(raw), ARG(partner_scores), ARG(norm_weight), ARG(norm_bias), ARG(hidden),
                                           ARG(mix), ARG(next_norm_weight), ARG(next_norm_bias), ARG(normalized)});
    require_position(position, device);
    const ReduceShape s = reduce_shape(raw, partner_scores);
    check_residual(s, hidden, mix);
    check_next_norm(s, normalized, next_norm_weight, next_norm_bias);
    const int param = same_dtype("norm parameter", {&norm_weight, &norm_bias});
    Launch launch(device);
    check(rlm_relation_norm_reduce(ptr(raw), f32(partner_scores), ptr(norm_weight), ptr(norm_bias), i64(position), nullptr,
                                   static_cast<float>(norm_eps), nullptr, f32(hidden), f32(mix), f32(next_norm_weight),
                                   f32(next_norm_bias), static_cast<float>(next_norm_eps), ptr(normalized), code(normalized), 1,
                                   0, nullptr, s.rows, s.k_out, s.dim, code(raw), param, launch.status, launch.stream));
}

void relation_norm_reduce_residual_norm_project(const Tensor& raw, const Tensor& partner_scores, const Tensor& norm_weight,
                                                const Tensor& norm_bias, const Tensor& position, double norm_eps,
                                                Tensor& hidden, const Tensor& mix, const Tensor& next_norm_weight,
                                                const Tensor& next_norm_bias, double next_norm_eps, Tensor& normalized,
                                                const Tensor& projection_weight, Tensor& projected) {
    const c10::Device device = contiguous({ARG(raw), ARG(partner_scores), ARG(norm_weight), ARG(norm_bias), ARG(hidden),
                                           ARG(mix), ARG(next_norm_weight), ARG(next_norm_bias), ARG(normalized),
                                           ARG(projection_weight), ARG(projected)});
    require_position(position, device);
    const ReduceShape s = reduce_shape(raw, partner_scores);
    check_residual(s, hidden, mix);
    check_next_norm(s, normalized, next_norm_weight, next_norm_bias);
    const int64_t n_out = projection_weight.size(0);
    TORCH_CHECK_VALUE(is_shape(projection_weight, {n_out, s.dim}) && is_shape(projected, {s.rows, n_out}) &&
                          projection_weight.scalar_type() == normalized.scalar_type() &&
                          projected.scalar_type() == normalized.scalar_type(),
                      "projection_weight must be [N, D] and projected [B, N] in the dtype of normalized");
    const int param = same_dtype("norm parameter", {&norm_weight, &norm_bias});
    Launch launch(device);
    check(rlm_relation_norm_reduce_project(ptr(raw), f32(partner_scores), ptr(norm_weight), ptr(norm_bias), i64(position),
                                           static_cast<float>(norm_eps), f32(hidden), f32(mix), f32(next_norm_weight),
                                           f32(next_norm_bias), static_cast<float>(next_norm_eps), ptr(normalized),
                                           ptr(projection_weight), ptr(projected), n_out, code(normalized), nullptr, s.rows,
                                           s.k_out, s.dim, code(raw), param, launch.status, launch.stream));
}

void slot_mix_residual(const Tensor& slot_context, const Tensor& anchor_active, const Tensor& slot_weight, const Tensor& gate,
                       Tensor& hidden) {
    const c10::Device device = contiguous({ARG(slot_context), ARG(anchor_active), ARG(slot_weight), ARG(gate), ARG(hidden)});
    TORCH_CHECK_VALUE(slot_context.dim() == 3, "slot_mix_residual: inconsistent shapes");
    const int64_t rows = slot_context.size(0), slots = slot_context.size(1), dim = slot_context.size(2);
    TORCH_CHECK_VALUE(is_shape(anchor_active, {rows, slots}) && slot_weight.numel() == slots && is_shape(hidden, {rows, dim}) &&
                          gate.numel() == 1,
                      "slot_mix_residual: inconsistent shapes");
    TORCH_CHECK_VALUE(anchor_active.scalar_type() == at::kBool || anchor_active.scalar_type() == at::kByte,
                      "anchor_active must be bool");
    for (const Named& a : {ARG(slot_context), ARG(slot_weight), ARG(gate), ARG(hidden)})
        TORCH_CHECK_VALUE(is_f32(*a.t), a.name, " must be float32");
    Launch launch(device);
    check(rlm_slot_mix_residual(f32(slot_context), static_cast<const uint8_t*>(anchor_active.data_ptr()), f32(slot_weight),
                                f32(gate), f32(hidden), rows, slots, dim, launch.stream));
}

using TailCall = decltype(&rlm_relation_layer_tail);

void layer_tail(TailCall launch_tail, const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                         const Tensor& partner_index, const Tensor& partner_scores, const Tensor& product_weight,
                         const Tensor& second_weight, const Tensor& second_bias, const Tensor& norm_weight,
                         const Tensor& norm_bias, const Tensor& position, double norm_eps, Tensor& hidden, const Tensor& mix,
                         const Tensor& next_norm_weight, const Tensor& next_norm_bias, double next_norm_eps,
                         Tensor& normalized, const OptTensor& query_weight, const OptTensor& query) {
    const c10::Device device = contiguous(
        {ARG(expanded_cache), ARG(operand_cache), ARG(anchor_index), ARG(partner_index), ARG(partner_scores),
         ARG(product_weight), ARG(second_weight), ARG(second_bias), ARG(norm_weight), ARG(norm_bias), ARG(hidden), ARG(mix),
         ARG(next_norm_weight), ARG(next_norm_bias), ARG(normalized), OPT(query_weight), OPT(query)});
    require_position(position, device);
    TORCH_CHECK_VALUE(operand_cache.dim() == 3 && partner_index.dim() == 2 && product_weight.dim() == 2 && second_weight.dim() == 2,
                      "relation_layer_tail: inconsistent shapes");
    const int64_t batch = operand_cache.size(0), max_t = operand_cache.size(1), rdim = operand_cache.size(2);
    const int64_t hdim = product_weight.size(0), dim = second_weight.size(0), k_out = partner_index.size(1);
    TORCH_CHECK_VALUE(is_shape(expanded_cache, {batch, max_t, 2 * hdim}) && is_shape(product_weight, {hdim, rdim}) &&
                          is_shape(second_weight, {dim, hdim}) && second_bias.numel() == dim && is_shape(anchor_index, {batch}) &&
                          is_shape(partner_index, {batch, k_out}) && is_shape(partner_scores, {batch, k_out}) &&
                          is_shape(hidden, {batch, dim}) && is_shape(normalized, {batch, dim}),
                      "relation_layer_tail: inconsistent shapes");
    TORCH_CHECK_VALUE(is_i32(anchor_index) && is_i32(partner_index), "index tensors must be int32");
    for (const Named& a : {ARG(partner_scores), ARG(hidden), ARG(mix), ARG(norm_weight), ARG(norm_bias), ARG(next_norm_weight),
                           ARG(next_norm_bias)})
        TORCH_CHECK_VALUE(is_f32(*a.t), a.name, " must be float32");
    int dtype = same_dtype("16-bit operand", {&expanded_cache, &operand_cache, &product_weight, &second_weight, &second_bias,
                                              &normalized});
    int64_t n_query = 0;
    if (query_weight.has_value()) {
        TORCH_CHECK_VALUE(query.has_value() && query_weight->dim() == 2 && query_weight->size(1) == dim &&
                              is_shape(*query, {batch, query_weight->size(0)}),
                          "query_weight [NQ, d] needs an output query [B, NQ]");
        n_query = query_weight->size(0);
        dtype = same_dtype("16-bit operand", {&expanded_cache, &*query_weight, &*query});
    }
    Launch launch(device);
    check(launch_tail(ptr(expanded_cache), ptr(operand_cache), i32(anchor_index), i32(partner_index),
                                  f32(partner_scores), ptr(product_weight), ptr(second_weight), ptr(second_bias),
                                  f32(norm_weight), f32(norm_bias), i64(position), static_cast<float>(norm_eps), f32(hidden),
                                  f32(mix), f32(next_norm_weight), f32(next_norm_bias), static_cast<float>(next_norm_eps),
                                  ptr(normalized), ptr(query_weight), ptr(query), batch, k_out, max_t, rdim, hdim, dim, n_query,
                                  dtype, launch.status, launch.stream));
}

#define TAIL_PARAMS                                                                                                      \
    const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,                                  \
        const Tensor &partner_index, const Tensor &partner_scores, const Tensor &product_weight,                          \
        const Tensor &second_weight, const Tensor &second_bias, const Tensor &norm_weight, const Tensor &norm_bias,      \
        const Tensor &position, double norm_eps, Tensor &hidden, const Tensor &mix, const Tensor &next_norm_weight,      \
        const Tensor &next_norm_bias, double next_norm_eps, Tensor &normalized, const OptTensor &query_weight,           \
        const OptTensor &query

void relation_layer_tail(TAIL_PARAMS) {
    layer_tail(&rlm_relation_layer_tail, expanded_cache, operand_cache, anchor_index, partner_index, partner_scores, product_weight, second_weight, second_bias,
               norm_weight, norm_bias, position, norm_eps, hidden, mix, next_norm_weight, next_norm_bias, next_norm_eps, normalized,
               query_weight, query);
}

void relation_layer_tail_wide(TAIL_PARAMS) {
    layer_tail(&rlm_relation_layer_tail_wide, expanded_cache, operand_cache, anchor_index, partner_index, partner_scores, product_weight, second_weight, second_bias,
               norm_weight, norm_bias, position, norm_eps, hidden, mix, next_norm_weight, next_norm_bias, next_norm_eps, normalized,
               query_weight, query);
}

void relation_mlp_rows(Tensor& out, const Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_index,
                       const Tensor& partner_index, const Tensor& partner_scores, const OptTensor& anchor_active,
                       const OptTensor& slot_weight, const OptTensor& scale, const Tensor& product_weight,
                       const Tensor& second_weight, const Tensor& second_bias, const Tensor& norm_weight,
                       const Tensor& norm_bias, double norm_eps, const OptTensor& residual, int64_t slots,
                       int64_t rows_per_seq, bool limit_by_position) {
    const c10::Device device = contiguous(
        {ARG(out), ARG(expanded_cache), ARG(operand_cache), ARG(anchor_index), ARG(partner_index), ARG(partner_scores),
         OPT(anchor_active), OPT(slot_weight), OPT(scale), ARG(product_weight), ARG(second_weight), ARG(second_bias),
         ARG(norm_weight), ARG(norm_bias), OPT(residual)});
    TORCH_CHECK_VALUE(out.dim() == 2 && operand_cache.dim() == 3 && product_weight.dim() == 2 && second_weight.dim() == 2 &&
                          partner_index.dim() >= 2 && slots >= 1 && rows_per_seq >= 1,
                      "relation_mlp_rows: inconsistent shapes");
    const int64_t rows = out.size(0), dim = out.size(1), n_seq = operand_cache.size(0), max_t = operand_cache.size(1);
    const int64_t rdim = operand_cache.size(2), hdim = product_weight.size(0), k_out = partner_index.size(-1);
    TORCH_CHECK_VALUE(is_shape(expanded_cache, {n_seq, max_t, 2 * hdim}) && is_shape(product_weight, {hdim, rdim}) &&
                          is_shape(second_weight, {dim, hdim}) && second_bias.numel() == dim && norm_weight.numel() == dim &&
                          norm_bias.numel() == dim && anchor_index.numel() == rows * slots &&
                          partner_index.numel() == rows * slots * k_out && partner_scores.numel() == rows * slots * k_out &&
                          n_seq * rows_per_seq == rows,
                      "relation_mlp_rows: inconsistent shapes");
    TORCH_CHECK_VALUE(is_i32(anchor_index) && is_i32(partner_index), "index tensors must be int32");
    for (const Named& a : {ARG(out), ARG(partner_scores), ARG(second_bias), ARG(norm_weight), ARG(norm_bias), OPT(slot_weight),
                           OPT(scale), OPT(residual)})
        TORCH_CHECK_VALUE(!a.t || is_f32(*a.t), a.name, " must be float32");
    TORCH_CHECK_VALUE((!residual.has_value() || residual->sizes() == out.sizes()) && (!scale.has_value() || scale->numel() == 1) &&
                          slot_weight.has_value() == anchor_active.has_value() &&
                          (!slot_weight.has_value() || (slot_weight->numel() == slots && anchor_active->numel() == rows * slots &&
                                                        anchor_active->element_size() == 1)),
                      "relation_mlp_rows: inconsistent shapes");
    const int dtype = same_dtype("16-bit operand", {&expanded_cache, &operand_cache, &product_weight, &second_weight});
    Launch launch(device);
    check(rlm_relation_mlp_rows(ptr(expanded_cache), ptr(operand_cache), i32(anchor_index), i32(partner_index),
                                f32(partner_scores), static_cast<const uint8_t*>(ptr(anchor_active)), f32(slot_weight),
                                f32(scale), ptr(product_weight), ptr(second_weight), f32(second_bias), f32(norm_weight),
                                f32(norm_bias), static_cast<float>(norm_eps), f32(residual), f32(out), rows, slots, n_seq,
                                rows_per_seq, max_t, rdim, hdim, dim, k_out, limit_by_position, dtype, launch.status,
                                launch.stream));
}

// ------------------------------------------------------------------ projections and the ends of a step

void check_projection(const Tensor& x, const Tensor& weight, const OptTensor& bias, c10::Device device) {
    contiguous({ARG(weight), OPT(bias)});
    TORCH_CHECK_VALUE(weight.device() == device && weight.dim() == 2 && weight.size(1) == x.size(1),
                      "weight must be [n_out, d_in] on the device of x");
    TORCH_CHECK_VALUE(x.scalar_type() == weight.scalar_type(), "x and weight must share one dtype");
    if (bias.has_value())
        TORCH_CHECK_VALUE(is_f32(*bias) && bias->numel() == weight.size(0), "bias must be float32 [n_out] on the device of x");
}

Tensor packed_projection(const Tensor& x, const Tensor& weight, const OptTensor& bias) {
    const c10::Device device = dense_rows({ARG(x)});
    check_projection(x, weight, bias, device);
    TORCH_CHECK_VALUE(x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf,
                      "packed_projection takes bfloat16 or float16 operands of one dtype");
    Launch launch(device);
    Tensor out = empty({x.size(0), weight.size(0)}, x.scalar_type(), device);
    check(rlm_packed_projection(ptr(x), x.stride(0), ptr(weight), f32(bias), ptr(out), x.size(0), x.size(1), weight.size(0),
                                code(x), code(out), 1, launch.status, launch.stream));
    return out;
}

void layer_norm_cast(const Tensor& x, const Tensor& norm_weight, const Tensor& norm_bias, double norm_eps, Tensor& out) {
    const c10::Device device = dense_rows({ARG(x)});
    contiguous({ARG(norm_weight), ARG(norm_bias), ARG(out)});
    TORCH_CHECK_VALUE(is_f32(x) && is_f32(norm_weight) && is_f32(norm_bias),
                      "layer_norm_cast takes fp32 rows and fp32 LayerNorm parameters");
    TORCH_CHECK_VALUE(out.sizes() == x.sizes() && norm_weight.numel() == x.size(1),
                      "out must have the shape of x and the norm parameters [d]");
    Launch launch(device);
    check(rlm_layer_norm_cast(f32(x), x.stride(0), f32(norm_weight), f32(norm_bias), static_cast<float>(norm_eps), ptr(out),
                              x.size(0), x.size(1), code(out), launch.stream));
}

Tensor decode_embed_norm(const Tensor& tokens, const Tensor& boundaries, const Tensor& token_table,
                         const Tensor& boundary_table, const Tensor& position_table, const Tensor& position, double scale,
                         const Tensor& norm1_weight, const Tensor& norm1_bias, Tensor& normalized1, const Tensor& norm2_weight,
                         const Tensor& norm2_bias, Tensor& normalized2, double norm_eps) {
    const c10::Device device = contiguous({ARG(tokens), ARG(boundaries), ARG(token_table), ARG(boundary_table),
                                           ARG(position_table), ARG(norm1_weight), ARG(norm1_bias), ARG(normalized1),
                                           ARG(norm2_weight), ARG(norm2_bias), ARG(normalized2)});
    require_position(position, device);
    TORCH_CHECK_VALUE(tokens.scalar_type() == at::kLong && boundaries.scalar_type() == at::kLong && is_f32(position_table),
                      "ids must be int64 and the position table float32");
    const int64_t batch = tokens.numel(), d_model = token_table.size(1);
    TORCH_CHECK_VALUE(boundaries.numel() == batch && boundary_table.size(1) == d_model && position_table.size(1) == d_model,
                      "decode_embed_norm: one boundary id per token and tables of one width");
    for (const Tensor* t : {&norm1_weight, &norm1_bias, &norm2_weight, &norm2_bias})
        TORCH_CHECK_VALUE(is_f32(*t) && t->numel() == d_model, "LayerNorm parameters must be float32 [d_model]");
    TORCH_CHECK_VALUE(is_shape(normalized1, {batch, d_model}) && is_shape(normalized2, {batch, d_model}) &&
                          normalized1.scalar_type() == normalized2.scalar_type(),
                      "normalized outputs must be [B, d_model] of one dtype");
    const int table = same_dtype("embedding table", {&token_table, &boundary_table});
    Launch launch(device);
    Tensor out = empty({batch, d_model}, at::kFloat, device);
    check(rlm_decode_embed(i64(tokens), i64(boundaries), ptr(token_table), ptr(boundary_table), f32(position_table),
                           i64(position), static_cast<float>(scale), f32(out), batch, d_model, token_table.size(0),
                           boundary_table.size(0), position_table.size(0), table, f32(norm1_weight), f32(norm1_bias),
                           ptr(normalized1), f32(norm2_weight), f32(norm2_bias), ptr(normalized2),
                           static_cast<float>(norm_eps), code(normalized1), launch.status, launch.stream));
    return out;
}

Two decode_front(const Tensor& tokens, const Tensor& boundaries, const Tensor& token_table, const Tensor& boundary_table,
                 const Tensor& position_table, const Tensor& position, double scale, const Tensor& norm1_weight,
                 const Tensor& norm1_bias, const Tensor& norm2_weight, const Tensor& norm2_bias, double norm_eps,
                 const Tensor& weight, int64_t n_first, Tensor& norm1_out, Tensor& norm2_out, Tensor& out_second) {
    const c10::Device device = contiguous({ARG(tokens), ARG(boundaries), ARG(token_table), ARG(boundary_table),
                                           ARG(position_table), ARG(norm1_weight), ARG(norm1_bias), ARG(norm2_weight),
                                           ARG(norm2_bias), ARG(weight), ARG(norm1_out), ARG(norm2_out), ARG(out_second)});
    require_position(position, device);
    TORCH_CHECK_VALUE(tokens.scalar_type() == at::kLong && boundaries.scalar_type() == at::kLong,
                      "token and boundary ids must be int64");
    TORCH_CHECK_VALUE(weight.dim() == 2 && token_table.dim() == 2, "decode_front: inconsistent shapes");
    const int64_t batch = tokens.numel(), d_model = token_table.size(1), n_total = weight.size(0);
    TORCH_CHECK_VALUE(boundaries.numel() == batch && boundary_table.size(1) == d_model && position_table.size(1) == d_model &&
                          weight.size(1) == d_model && n_first > 0 && n_first < n_total &&
                          is_shape(norm1_out, {batch, d_model}) && is_shape(norm2_out, {batch, d_model}) &&
                          is_shape(out_second, {batch, n_total - n_first}),
                      "decode_front: inconsistent shapes");
    TORCH_CHECK_VALUE(is_f32(position_table), "position_table must be float32 of the model width");
    for (const Named& a : {ARG(norm1_weight), ARG(norm1_bias), ARG(norm2_weight), ARG(norm2_bias)})
        TORCH_CHECK_VALUE(is_f32(*a.t) && a.t->numel() == d_model, a.name, " must be float32 of the model width");
    const int dtype = same_dtype("16-bit operand", {&token_table, &boundary_table, &weight, &norm1_out, &norm2_out, &out_second});
    Launch launch(device);
    Tensor hidden = empty({batch, d_model}, at::kFloat, device), first = empty({batch, n_first}, weight.scalar_type(), device);
    check(rlm_decode_front(i64(tokens), i64(boundaries), ptr(token_table), ptr(boundary_table), f32(position_table),
                           i64(position), static_cast<float>(scale), f32(norm1_weight), f32(norm1_bias), f32(norm2_weight),
                           f32(norm2_bias), static_cast<float>(norm_eps), ptr(weight), f32(hidden), ptr(norm1_out),
                           ptr(norm2_out), ptr(first), ptr(out_second), batch, d_model, n_first, n_total - n_first,
                           token_table.size(0), boundary_table.size(0), position_table.size(0), dtype, launch.status,
                           launch.stream));
    return {hidden, first};
}

Tensor greedy_token(const Tensor& logits, int64_t vocab, const OptTensor& position) {
    const c10::Device device = dense_rows({ARG(logits)});
    TORCH_CHECK_VALUE(vocab >= 1 && vocab <= logits.size(1), "logits must be [rows, >= vocab]");
    if (position.has_value()) require_position(*position, device);
    Launch launch(device);
    Tensor out = empty({logits.size(0)}, at::kLong, device);
    check(rlm_greedy_token(ptr(logits), logits.stride(0), i64(out), position.has_value() ? i64(*position) : nullptr,
                           logits.size(0), vocab, code(logits), launch.stream));
    return out;
}

void few_rows(Tensor& out, Tensor* out2, const Tensor& x, const Tensor& weight, const Tensor* weight2, const OptTensor& bias,
              const OptTensor& bias2) {
    const c10::Device device = dense_rows({ARG(x)});
    TORCH_CHECK_VALUE(contiguous({ARG(out), ARG(weight), Named{"out2", out2}, Named{"weight2", weight2}, OPT(bias), OPT(bias2)}) == device,
                      "weights and results must be on the device of x");
    const auto fits = [&](const Tensor& o, const Tensor& w, const OptTensor& b) {
        TORCH_CHECK_VALUE(is_f32(x) && is_f32(w) && is_f32(o) && (!b.has_value() || is_f32(*b)), "few_rows_projection takes float32 tensors");
        TORCH_CHECK_VALUE(w.dim() == 2 && w.size(1) == x.size(1) && is_shape(o, {x.size(0), w.size(0)}) &&
                              (!b.has_value() || b->numel() == w.size(0)),
                          "few_rows_projection: weight [n, d], bias [n], result [rows, n]");
    };
    fits(out, weight, bias);
    if (out2) fits(*out2, *weight2, bias2);
    Launch launch(device);
    check(rlm_few_rows_projection(f32(x), x.stride(0), f32(weight), f32(bias), f32(out), weight2 ? f32(*weight2) : nullptr, f32(bias2),
                                  out2 ? f32(*out2) : nullptr, x.size(0), x.size(1), weight.size(0), weight2 ? weight2->size(0) : 0,
                                  launch.stream));
}

void few_rows_projection(Tensor& out, const Tensor& x, const Tensor& weight, const OptTensor& bias) {
    few_rows(out, nullptr, x, weight, nullptr, bias, std::nullopt);
}

void few_rows_projection_pair(Tensor& out, Tensor& out2, const Tensor& x, const Tensor& weight, const Tensor& weight2,
                              const OptTensor& bias2) {
    few_rows(out, &out2, x, weight, &weight2, std::nullopt, bias2);
}

Tensor skinny_projection(const Tensor& x, const Tensor& weight, const OptTensor& bias) {
    const c10::Device device = dense_rows({ARG(x)});
    check_projection(x, weight, bias, device);
    Launch launch(device);
    Tensor out = empty({x.size(0), weight.size(0)}, x.scalar_type(), device);
    check(rlm_skinny_projection(ptr(x), x.stride(0), ptr(weight), f32(bias), ptr(out), x.size(0), x.size(1), weight.size(0),
                                code(x), 0, nullptr, nullptr, nullptr, launch.stream));
    return out;
}

Tensor skinny_greedy(const Tensor& x, const Tensor& weight, const OptTensor& bias, int64_t vocab, Tensor& scratch,
                     const OptTensor& position, const Tensor& next_token, c10::Device device) {
    check_projection(x, weight, bias, device);
    contiguous({ARG(scratch), ARG(next_token)});
    TORCH_CHECK_VALUE(scratch.scalar_type() == at::kByte && scratch.numel() >= rlm_skinny_argmax_scratch_bytes(),
                      "scratch must be a uint8 tensor of skinny_argmax_scratch_bytes() bytes");
    TORCH_CHECK_VALUE(vocab >= 1 && vocab <= weight.size(0), "vocab must lie within the projection's outputs");
    TORCH_CHECK_VALUE(next_token.scalar_type() == at::kLong && is_shape(next_token, {x.size(0)}),
                      "next_token must be int64 [rows]");
    if (position.has_value()) require_position(*position, device);
    Launch launch(device);
    Tensor out = empty({x.size(0), weight.size(0)}, x.scalar_type(), device);
    check(rlm_skinny_projection(ptr(x), x.stride(0), ptr(weight), f32(bias), ptr(out), x.size(0), x.size(1), weight.size(0),
                                code(x), vocab, ptr(scratch), i64(next_token),
                                position.has_value() ? i64(*position) : nullptr, launch.stream));
    return out;
}

Two skinny_projection_greedy(const Tensor& x, const Tensor& weight, const OptTensor& bias, int64_t vocab, Tensor& scratch,
                             const OptTensor& position) {
    const c10::Device device = dense_rows({ARG(x)});
    Tensor next = empty({x.size(0)}, at::kLong, device);
    Tensor out = skinny_greedy(x, weight, bias, vocab, scratch, position, next, device);
    return {out, next};
}

Tensor skinny_projection_greedy_into(const Tensor& x, const Tensor& weight, const OptTensor& bias, int64_t vocab,
                                     Tensor& scratch, const OptTensor& position, Tensor& next_token) {
    return skinny_greedy(x, weight, bias, vocab, scratch, position, next_token, dense_rows({ARG(x)}));
}

// ------------------------------------------------------------------ the single-precision step in three calls
//
// A step without a captured graph is bound by the host: ten operator calls of 4-5 us each for one layer, whose kernels
// take 42 us.  These are the same operators in the same order, a call for what comes before the layers, one per layer and
// one for the heads; they exist as extension functions only, and where those decline the step makes its calls one by one.

Tensor single_precision_front(const Tensor& tokens, const Tensor& boundaries, const Tensor& token_table, const Tensor& boundary_table,
                              const Tensor& position_table, const Tensor& position, double scale, const Tensor& memory_norm_w,
                              const Tensor& memory_norm_b, Tensor& memory_rows, const Tensor& input_norm_w,
                              const Tensor& input_norm_b, Tensor& normalized, double norm_eps, Tensor& packed,
                              const Tensor& packed_weight, Tensor& anchor_keys, Tensor& partner_keys, Tensor& operand_cache,
                              Tensor& partner_anchor_cache, ROUTER_PARAMS, int64_t block_size) {
    Tensor hidden = decode_embed_norm(tokens, boundaries, token_table, boundary_table, position_table, position, scale, memory_norm_w,
                                      memory_norm_b, memory_rows, input_norm_w, input_norm_b, normalized, norm_eps);
    few_rows_projection(packed, memory_rows, packed_weight, std::nullopt);
    sparse_cache_append(packed, anchor_keys, partner_keys, operand_cache, partner_anchor_cache, ROUTER_VALUES, position, block_size);
    return hidden;
}

Two single_precision_layer(const Tensor& normalized, const Tensor& query_weight, Tensor& query, SELECT_PARAMS, const Tensor& position,
                           int64_t local_window, int64_t top_blocks, int64_t k_out, bool strict_valid, Tensor& relation_hidden,
                           Tensor& expanded_cache, const Tensor& operand_cache, const Tensor& anchor_weight,
                           const Tensor& partner_weight, const Tensor& product_weight, const Tensor& first_bias,
                           Tensor& second_rows, const Tensor& second_weight, const Tensor& second_bias, const Tensor& norm_weight,
                           const Tensor& norm_bias, double norm_eps, Tensor& hidden, const Tensor& mix,
                           const Tensor& next_norm_weight, const Tensor& next_norm_bias, Tensor& next_normalized) {
    few_rows_projection(query, normalized, query_weight, std::nullopt);
    auto [anchor, anchor_score, partner, score] =
        select(SELECT_TENSORS, &position, nullptr, nullptr, local_window, top_blocks, k_out, strict_valid);
    relation_hidden_cache_update_out(relation_hidden, expanded_cache, operand_cache, anchor, partner, anchor_weight, partner_weight,
                                     product_weight, first_bias, position);
    Tensor rows = second_rows.view({-1, second_weight.size(0)});
    few_rows_projection(rows, relation_hidden.view({-1, second_weight.size(1)}), second_weight, second_bias);
    relation_norm_reduce_residual_norm(second_rows, score, norm_weight, norm_bias, position, norm_eps, hidden, mix, next_norm_weight,
                                       next_norm_bias, norm_eps, next_normalized);
    return {anchor, partner};
}

Two single_precision_heads(const Tensor& normalized, const Tensor& token_weight, const Tensor& boundary_weight, const Tensor& boundary_bias,
                           Tensor& position) {
    const c10::Device device = dense_rows({ARG(normalized)});
    Tensor tokens = empty({normalized.size(0), token_weight.size(0)}, at::kFloat, device);
    Tensor boundaries = empty({normalized.size(0), boundary_weight.size(0)}, at::kFloat, device);
    few_rows_projection_pair(tokens, boundaries, normalized, token_weight, boundary_weight, boundary_bias);
    at::AutoDispatchBelowADInplaceOrView below;          // (the version counter is advanced by the caller)
    position.add_(1);
    return {tokens, boundaries};
}

// ------------------------------------------------------------------ a whole-sequence layer, its operators in two groups
//
// One after the other from Python a short prompt's eight launches took the host longer than the device.

// The state of sequences x [B, T, d]: what sequence_state leaves, the expanded cache, the packed rows.
std::vector<Tensor> prefill_state(const Tensor& x, const Tensor& norm_weight, const Tensor& norm_bias, double norm_eps,
                                  const Tensor& packed_weight, int64_t relation_dim, int64_t block_size,
                                  const Tensor& anchor_conv_weight, const Tensor& partner_conv_weight,
                                  const Tensor& expand_weight, const Tensor& expand_bias) {
    const int64_t batch = x.size(0), length = x.size(1);
    const Tensor rows = x.view({batch * length, x.size(2)});
    Tensor memory = empty(rows.sizes(), packed_weight.scalar_type(), x.device());
    layer_norm_cast(rows, norm_weight, norm_bias, norm_eps, memory);
    const Tensor packed = packed_projection(memory, packed_weight, std::nullopt).view({batch, length, packed_weight.size(0)});
    std::vector<Tensor> state = sequence_state(packed, 0, relation_dim, block_size, anchor_conv_weight, partner_conv_weight);
    state.push_back(packed_projection(state[2].view({batch * length, relation_dim}), expand_weight, expand_bias)
                        .view({batch, length, expand_weight.size(0)}));
    state.push_back(packed);
    return state;
}

// The layer's output [B, T, d] for residual inputs x and their state; where the selector's tile does not fit, none, and the
// queries, which then go on to the selector of rows.
std::vector<Tensor> prefill_layer(const Tensor& x, const Tensor& norm_weight, const Tensor& norm_bias, double norm_eps, const Tensor& query_weight,
                     const Tensor& anchor_keys, const Tensor& anchor_mean, const Tensor& anchor_std, const Tensor& anchor_gamma,
                     const Tensor& anchor_bias, const Tensor& partner_anchor_cache, const Tensor& partner_keys,
                     const Tensor& partner_mean, const Tensor& partner_std, const Tensor& partner_gamma, const Tensor& partner_bias,
                     int64_t local_window, int64_t top_blocks, int64_t k_out, bool strict_valid, const Tensor& expanded_cache,
                     const Tensor& operand_cache, const Tensor& mix, const Tensor& product_weight, const Tensor& second_weight,
                     const Tensor& second_bias, const Tensor& relation_norm_weight, const Tensor& relation_norm_bias) {
    const int64_t batch = x.size(0), length = x.size(1), dim = x.size(2);
    const Tensor rows = x.view({batch * length, dim});
    Tensor normalized = empty(rows.sizes(), query_weight.scalar_type(), x.device());
    layer_norm_cast(rows, norm_weight, norm_bias, norm_eps, normalized);
    const Tensor q = packed_projection(normalized, query_weight, std::nullopt);
    const Tensor anchor_query = q.narrow(1, 0, 64), router_query = q.narrow(1, 64, 64), partner_base = q.narrow(1, 128, 128);
    bool fits = true;
    const auto [anchor, anchor_score, partner, score] = select_prefill(
        {anchor_query, anchor_keys, router_query, anchor_mean, anchor_std, anchor_gamma, anchor_bias, partner_base, partner_anchor_cache,
         partner_keys, partner_mean, partner_std, partner_gamma, partner_bias},
        length, local_window, top_blocks, k_out, strict_valid, &fits);
    if (!fits) return {Tensor(), q};
    Tensor out = empty(rows.sizes(), at::kFloat, x.device());
    relation_mlp_rows(out, expanded_cache, operand_cache, anchor, partner, score, std::nullopt, std::nullopt, mix, product_weight,
                      second_weight, second_bias, relation_norm_weight, relation_norm_bias, norm_eps, rows.contiguous(), 1, length, true);
    return {out.view({batch, length, dim})};
}

// ------------------------------------------------------------------ what surrounds an operator

using Stack = torch::jit::Stack;

template <typename F>
void for_each_tensor(const c10::IValue& v, F&& f) {
    if (v.isTensor()) {
        f(v.toTensor());
    } else if (v.isTensorList()) {
        for (const Tensor& t : v.toTensorList().vec()) f(t);
    }
}

// Derivatives are not implemented: in grad mode floating-point results of arguments that require one carry a node that
// raises when it is asked for it.  Arguments that are written stay as they are, a leaf included.  (PyTorch's own
// fallback for such operators refuses to write a leaf that requires a derivative, and any forward-mode tangent.)
void no_derivative(const c10::OperatorHandle& op, c10::DispatchKeySet keys, Stack* stack) {
    const c10::FunctionSchema& schema = op.schema();
    torch::autograd::variable_list inputs;
    if (at::GradMode::is_enabled())
        for (const c10::IValue& v : torch::jit::last(*stack, schema.arguments().size()))
            for_each_tensor(v, [&](const Tensor& t) {
                if (t.defined() && t.requires_grad()) inputs.push_back(t);
            });
    {
        at::AutoDispatchBelowAutograd below;
        op.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
    }
    if (inputs.empty() || schema.returns().empty()) return;
    const auto node = std::make_shared<torch::autograd::NotImplemented>(schema.name());
    node->set_next_edges(torch::autograd::collect_next_edges(inputs));
    for (const c10::IValue& v : torch::jit::last(*stack, schema.returns().size()))
        for_each_tensor(v, [&](const Tensor& t) {
            if (t.defined() && torch::autograd::isDifferentiableType(t.scalar_type())) torch::autograd::set_history(t, node);
        });
}

// The version counters of the arguments that the schema marks as written advance.
void bump_versions(const c10::OperatorHandle& op, c10::DispatchKeySet keys, Stack* stack) {
    const auto& arguments = op.schema().arguments();
    std::vector<Tensor> written;
    const auto values = torch::jit::last(*stack, arguments.size());
    for (size_t i = 0; i < arguments.size(); ++i)
        if (arguments[i].alias_info() && arguments[i].alias_info()->isWrite())
            for_each_tensor(values[i], [&](const Tensor& t) {
                if (t.defined() && !t.is_inference()) written.push_back(t);
            });
    {
        at::AutoDispatchBelowADInplaceOrView below;
        op.redispatchBoxed(keys & c10::after_ADInplaceOrView_keyset, stack);
    }
    for (const Tensor& t : written) t.unsafeGetTensorImpl()->bump_version();
}

Tensor status_word_of(int64_t device_index) { return status_word(static_cast<int>(device_index)); }

}  // namespace

// ------------------------------------------------------------------ registration

#define SELECT_SCHEMA                                                                                                    \
    "Tensor anchor_query, Tensor anchor_keys, Tensor anchor_router_query, Tensor anchor_block_mean, "                    \
    "Tensor anchor_block_std, Tensor anchor_gamma, Tensor anchor_bias, Tensor partner_base, "                            \
    "Tensor partner_anchor_cache, Tensor partner_keys, Tensor partner_block_mean, Tensor partner_block_std, "            \
    "Tensor partner_gamma, Tensor partner_bias, "

// Every operator with its schema, its implementation and what surrounds it (above); with `MUTATES`, arguments that
// are written.
#define FOR_EACH_OP(PURE, MUTATES)                                                                                       \
    PURE(relation_select_packed, "(" SELECT_SCHEMA "Tensor position, SymInt local_window, SymInt top_blocks, "           \
         "SymInt k_out, bool strict_valid) -> (Tensor, Tensor, Tensor, Tensor)")                                         \
    PURE(relation_select_packed_rows, "(" SELECT_SCHEMA "Tensor row_batch, Tensor row_position, SymInt local_window, "   \
         "SymInt top_blocks, SymInt k_out, bool strict_valid) -> (Tensor, Tensor, Tensor, Tensor)")                      \
    PURE(relation_select_packed_prefill, "(" SELECT_SCHEMA "SymInt query_length, SymInt local_window, "                  \
         "SymInt top_blocks, SymInt k_out, bool strict_valid) -> (Tensor, Tensor, Tensor, Tensor)")                      \
    PURE(relation_select_multi_rows, "(" SELECT_SCHEMA "Tensor row_batch, Tensor row_position, SymInt local_window, "    \
         "SymInt top_blocks, SymInt partners_per_anchor, bool strict_valid) -> "                                         \
         "(Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)")                                                             \
    PURE(relation_select_multi_prefill, "(" SELECT_SCHEMA "SymInt query_length, SymInt local_window, "                   \
         "SymInt top_blocks, SymInt partners_per_anchor, bool strict_valid) -> "                                         \
         "(Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)")                                                             \
    PURE(relation_select_multi_prefill_scores, "(" SELECT_SCHEMA "SymInt query_length, SymInt local_window, "            \
         "SymInt top_blocks, SymInt partners_per_anchor, bool strict_valid) -> "                                         \
         "(Tensor, Tensor, Tensor, Tensor, Tensor)")                                                                     \
    MUTATES(router_cache_update,                                                                                         \
            "(Tensor anchor_raw, Tensor partner_raw, Tensor(a2!) anchor_raw_cache, Tensor(a3!) partner_raw_cache, "      \
            "Tensor(a4!) anchor_conv_cache, Tensor(a5!) partner_conv_cache, Tensor(a6!) anchor_mean, "                   \
            "Tensor(a7!) anchor_std, Tensor(a8!) partner_mean, Tensor(a9!) partner_std, Tensor anchor_conv_weight, "     \
            "Tensor partner_conv_weight, Tensor position, SymInt block_size) -> Tensor")                                 \
    MUTATES(sparse_cache_append,                                                                                         \
            "(Tensor packed, Tensor(a1!) anchor_keys, Tensor(a2!) partner_keys, Tensor(a3!) operand_cache, "             \
            "Tensor(a4!) partner_anchor_cache, Tensor(a5!) anchor_raw_cache, Tensor(a6!) partner_raw_cache, "            \
            "Tensor(a7!) anchor_conv_cache, Tensor(a8!) partner_conv_cache, Tensor(a9!) anchor_mean, "                   \
            "Tensor(a10!) anchor_std, Tensor(a11!) partner_mean, Tensor(a12!) partner_std, Tensor anchor_conv_weight, "  \
            "Tensor partner_conv_weight, Tensor position, SymInt block_size) -> ()")                                     \
    MUTATES(router_cache_prefill,                                                                                        \
            "(Tensor anchor_raw, Tensor partner_raw, Tensor(a2!) anchor_raw_cache, Tensor(a3!) partner_raw_cache, "      \
            "Tensor(a4!) anchor_conv_cache, Tensor(a5!) partner_conv_cache, Tensor(a6!) anchor_mean, "                   \
            "Tensor(a7!) anchor_std, Tensor(a8!) partner_mean, Tensor(a9!) partner_std, Tensor anchor_conv_weight, "     \
            "Tensor partner_conv_weight, SymInt block_size) -> ()")                                                      \
    PURE(sequence_state, "(Tensor packed, SymInt slots, SymInt relation_dim, SymInt block_size, "                        \
         "Tensor anchor_conv_weight, Tensor partner_conv_weight) -> Tensor[]")                                           \
    PURE(relation_hidden_cached, "(Tensor expanded_cache, Tensor operand_cache, Tensor anchor_index, "                   \
         "Tensor partner_index, Tensor product_weight) -> Tensor")                                                       \
    MUTATES(relation_hidden_cached_out, "(Tensor(a0!) out, Tensor expanded_cache, Tensor operand_cache, "                \
            "Tensor anchor_index, Tensor partner_index, Tensor product_weight) -> ()")                                   \
    PURE(relation_hidden_cached_rows, "(Tensor expanded_cache, Tensor operand_cache, Tensor anchor_index, "              \
         "Tensor partner_index, Tensor product_weight, Tensor row_batch) -> Tensor")                                     \
    MUTATES(relation_hidden_cached_rows_out, "(Tensor(a0!) out, Tensor expanded_cache, Tensor operand_cache, "           \
            "Tensor anchor_index, Tensor partner_index, Tensor product_weight, Tensor row_batch) -> ()")                 \
    MUTATES(relation_hidden_cache_update, "(Tensor(a0!) expanded_cache, Tensor operand_cache, Tensor anchor_index, "     \
            "Tensor partner_index, Tensor anchor_weight, Tensor partner_weight, Tensor product_weight, "                 \
            "Tensor first_bias, Tensor position) -> Tensor")                                                             \
    MUTATES(relation_hidden_cache_update_out, "(Tensor(a0!) out, Tensor(a1!) expanded_cache, Tensor operand_cache, "     \
            "Tensor anchor_index, Tensor partner_index, Tensor anchor_weight, Tensor partner_weight, "                   \
            "Tensor product_weight, Tensor first_bias, Tensor position) -> ()")                                          \
    MUTATES(expanded_cache_append, "(Tensor(a0!) expanded_cache, Tensor operand_cache, Tensor anchor_weight, "           \
            "Tensor partner_weight, Tensor first_bias, Tensor position) -> ()")                                          \
    MUTATES(expanded_cache_append_packed, "(Tensor(a0!) expanded_cache, Tensor packed, Tensor anchor_weight, "           \
            "Tensor partner_weight, Tensor first_bias, Tensor position) -> ()")                                          \
    PURE(relation_norm_reduce, "(Tensor raw, Tensor partner_scores, Tensor norm_weight, Tensor norm_bias, "              \
         "Tensor position, float norm_eps) -> Tensor")                                                                   \
    PURE(relation_norm_reduce_rows, "(Tensor raw, Tensor partner_scores, Tensor norm_weight, Tensor norm_bias, "         \
         "Tensor row_position, float norm_eps) -> Tensor")                                                               \
    MUTATES(relation_norm_reduce_residual, "(Tensor raw, Tensor partner_scores, Tensor norm_weight, "                    \
            "Tensor norm_bias, Tensor position, float norm_eps, Tensor(a6!) hidden, Tensor mix) -> ()")                  \
    MUTATES(relation_norm_reduce_residual_norm, "(Tensor raw, Tensor partner_scores, Tensor norm_weight, "               \
            "Tensor norm_bias, Tensor position, float norm_eps, Tensor(a6!) hidden, Tensor mix, "                        \
            "Tensor next_norm_weight, Tensor next_norm_bias, float next_norm_eps, Tensor(a11!) normalized) -> ()")       \
    MUTATES(relation_norm_reduce_residual_norm_project, "(Tensor raw, Tensor partner_scores, Tensor norm_weight, "       \
            "Tensor norm_bias, Tensor position, float norm_eps, Tensor(a6!) hidden, Tensor mix, "                        \
            "Tensor next_norm_weight, Tensor next_norm_bias, float next_norm_eps, Tensor(a11!) normalized, "             \
            "Tensor projection_weight, Tensor(a13!) projected) -> ()")                                                   \
    MUTATES(slot_mix_residual, "(Tensor slot_context, Tensor anchor_active, Tensor slot_weight, Tensor gate, "           \
            "Tensor(a4!) hidden) -> ()")                                                                                 \
    MUTATES(relation_layer_tail, "(Tensor expanded_cache, Tensor operand_cache, Tensor anchor_index, "                   \
            "Tensor partner_index, Tensor partner_scores, Tensor product_weight, Tensor second_weight, "                 \
            "Tensor second_bias, Tensor norm_weight, Tensor norm_bias, Tensor position, float norm_eps, "                \
            "Tensor(a12!) hidden, Tensor mix, Tensor next_norm_weight, Tensor next_norm_bias, float next_norm_eps, "     \
            "Tensor(a17!) normalized, Tensor? query_weight, Tensor(a19!)? query) -> ()")                                 \
    MUTATES(relation_layer_tail_wide, "(Tensor expanded_cache, Tensor operand_cache, Tensor anchor_index, "              \
            "Tensor partner_index, Tensor partner_scores, Tensor product_weight, Tensor second_weight, "                 \
            "Tensor second_bias, Tensor norm_weight, Tensor norm_bias, Tensor position, float norm_eps, "                \
            "Tensor(a12!) hidden, Tensor mix, Tensor next_norm_weight, Tensor next_norm_bias, float next_norm_eps, "     \
            "Tensor(a17!) normalized, Tensor? query_weight, Tensor(a19!)? query) -> ()")                                 \
    MUTATES(relation_mlp_rows, "(Tensor(a0!) out, Tensor expanded_cache, Tensor operand_cache, Tensor anchor_index, "     \
            "Tensor partner_index, Tensor partner_scores, Tensor? anchor_active, Tensor? slot_weight, Tensor? scale, "   \
            "Tensor product_weight, Tensor second_weight, Tensor second_bias, Tensor norm_weight, Tensor norm_bias, "    \
            "float norm_eps, Tensor? residual, SymInt slots, SymInt rows_per_seq, bool limit_by_position) -> ()")        \
    PURE(packed_projection, "(Tensor x, Tensor weight, Tensor? bias=None) -> Tensor")                                    \
    MUTATES(layer_norm_cast, "(Tensor x, Tensor norm_weight, Tensor norm_bias, float norm_eps, Tensor(a4!) out) -> ()")  \
    MUTATES(decode_embed_norm, "(Tensor tokens, Tensor boundaries, Tensor token_table, Tensor boundary_table, "          \
            "Tensor position_table, Tensor position, float scale, Tensor norm1_weight, Tensor norm1_bias, "              \
            "Tensor(a9!) normalized1, Tensor norm2_weight, Tensor norm2_bias, Tensor(a12!) normalized2, "                \
            "float norm_eps) -> Tensor")                                                                                 \
    MUTATES(decode_front, "(Tensor tokens, Tensor boundaries, Tensor token_table, Tensor boundary_table, "               \
            "Tensor position_table, Tensor position, float scale, Tensor norm1_weight, Tensor norm1_bias, "              \
            "Tensor norm2_weight, Tensor norm2_bias, float norm_eps, Tensor weight, SymInt n_first, "                    \
            "Tensor(a14!) norm1_out, Tensor(a15!) norm2_out, Tensor(a16!) out_second) -> (Tensor, Tensor)")              \
    MUTATES(greedy_token, "(Tensor logits, SymInt vocab, Tensor(a2!)? position) -> Tensor")                              \
    MUTATES(few_rows_projection, "(Tensor(a0!) out, Tensor x, Tensor weight, Tensor? bias=None) -> ()")                  \
    MUTATES(few_rows_projection_pair, "(Tensor(a0!) out, Tensor(a1!) out2, Tensor x, Tensor weight, Tensor weight2, "     \
            "Tensor? bias2=None) -> ()")                                                                                 \
    PURE(skinny_projection, "(Tensor x, Tensor weight, Tensor? bias=None) -> Tensor")                                    \
    MUTATES(skinny_projection_greedy, "(Tensor x, Tensor weight, Tensor? bias, SymInt vocab, Tensor(a4!) scratch, "      \
            "Tensor(a5!)? position) -> (Tensor, Tensor)")                                                                \
    MUTATES(skinny_projection_greedy_into, "(Tensor x, Tensor weight, Tensor? bias, SymInt vocab, "                      \
            "Tensor(a4!) scratch, Tensor(a5!)? position, Tensor(a6!) next_token) -> Tensor")

#define DEFINE(name, schema) m.def(#name schema, {at::Tag::pt2_compliant_tag});
#define IMPLEMENT(name, schema) m.impl(#name, TORCH_FN(name));
#define NO_DERIVATIVE(name, schema) m.impl(#name, torch::CppFunction::makeFromBoxedFunction<&no_derivative>());
#define BUMP_VERSIONS(name, schema) m.impl(#name, torch::CppFunction::makeFromBoxedFunction<&bump_versions>());
#define NOTHING(name, schema)

TORCH_LIBRARY_FRAGMENT(relation_lm, m) {
    FOR_EACH_OP(DEFINE, DEFINE)
    m.def("_status_word(int device_index) -> Tensor", &status_word_of);
}
TORCH_LIBRARY_IMPL(relation_lm, CUDA, m) { FOR_EACH_OP(IMPLEMENT, IMPLEMENT) }
TORCH_LIBRARY_IMPL(relation_lm, Autograd, m) { FOR_EACH_OP(NO_DERIVATIVE, NO_DERIVATIVE) }
TORCH_LIBRARY_IMPL(relation_lm, ADInplaceOrView, m) { FOR_EACH_OP(NOTHING, BUMP_VERSIONS) }

#define FOR_EACH_LEX_OP(PURE)                                                                                            \
    PURE(anchor_select, "(Tensor anchor_query, Tensor anchor_keys, Tensor router_query, Tensor block_mean, "             \
         "Tensor block_std, Tensor gamma, Tensor bias, Tensor position, SymInt local_window, SymInt top_blocks, "        \
         "bool strict_valid) -> (Tensor, Tensor)")                                                                       \
    PURE(partner_topk, "(Tensor partner_query, Tensor partner_keys, Tensor router_query, Tensor block_mean, "            \
         "Tensor block_std, Tensor gamma, Tensor bias, Tensor position, Tensor anchor_index, SymInt local_window, "      \
         "SymInt top_blocks, SymInt k_out, bool strict_valid) -> (Tensor, Tensor)")

TORCH_LIBRARY_FRAGMENT(relationlex, m) { FOR_EACH_LEX_OP(DEFINE) }
TORCH_LIBRARY_IMPL(relationlex, CUDA, m) { FOR_EACH_LEX_OP(IMPLEMENT) }
TORCH_LIBRARY_IMPL(relationlex, Autograd, m) { FOR_EACH_LEX_OP(NO_DERIVATIVE) }

// ------------------------------------------------------------------ direct calls from Python
//
// An operator call through the dispatcher costs the host 2-4 us (boxing twenty arguments, the autograd and
// version-counter fallbacks), as much as its launch, and the passes of a small model are bound by exactly that.
// Each operator is therefore a plain extension function too.  It returns NotImplemented, and the caller takes the
// dispatcher, whenever the dispatcher would have anything to do: arguments that are not plain CUDA tensors (views that
// are still to be negated, tensors of zeros without memory and the like among them), a derivative to record, a mode, a
// tracer, a transform or a profiler at work.
namespace {

using c10::DispatchKey;
using c10::DispatchKeySet;

constexpr DispatchKeySet kInterposing({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::PythonDispatcher,
                                       DispatchKey::PreDispatch, DispatchKey::Functionalize, DispatchKey::Tracer,
                                       DispatchKey::Batched, DispatchKey::VmapMode, DispatchKey::FuncTorchBatched,
                                       DispatchKey::FuncTorchVmapMode, DispatchKey::FuncTorchGradWrapper,
                                       DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode,
                                       DispatchKey::FuncTorchBatchedDecomposition, DispatchKey::Negative, DispatchKey::Conjugate,
                                       DispatchKey::ZeroTensor, DispatchKey::Sparse, DispatchKey::SparseCsr,
                                       DispatchKey::Quantized, DispatchKey::NestedTensor, DispatchKey::TESTING_ONLY_GenericWrapper,
                                       DispatchKey::TESTING_ONLY_GenericMode});

bool nothing_interposed() {
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(kInterposing) && !at::impl::torch_function_mode_enabled() &&
           !at::hasThreadLocalCallbacks() && !at::hasGlobalCallbacks();
}

const Tensor* plain_tensor(PyObject* o, bool grad) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.key_set().has_any(kInterposing) || t.is_inference() || (grad && t.requires_grad())) return nullptr;
    return &t;
}

// An argument on its way from Python: load() says whether it is of the plain kind.
template <typename T> struct Arg;
template <> struct Arg<const Tensor&> {
    const Tensor* t;
    bool load(PyObject* o, bool grad) { return (t = plain_tensor(o, grad)) != nullptr; }
    const Tensor& get() { return *t; }
    void written() {}
};
template <> struct Arg<Tensor&> {
    Tensor t;
    bool load(PyObject* o, bool grad) {
        const Tensor* p = plain_tensor(o, grad);
        if (p) t = *p;
        return p != nullptr;
    }
    Tensor& get() { return t; }
    void written() { t.unsafeGetTensorImpl()->bump_version(); }
};
template <> struct Arg<const OptTensor&> {
    OptTensor t;
    bool load(PyObject* o, bool grad) {
        if (o == Py_None) return true;
        const Tensor* p = plain_tensor(o, grad);
        if (p) t = *p;
        return p != nullptr;
    }
    const OptTensor& get() { return t; }
    void written() {}
};
template <> struct Arg<int64_t> {
    int64_t v;
    bool load(PyObject* o, bool) {
        if (!PyLong_CheckExact(o)) return false;
        v = PyLong_AsLongLong(o);
        if (v != -1 || !PyErr_Occurred()) return true;
        PyErr_Clear();
        return false;
    }
    int64_t get() { return v; }
    void written() {}
};
template <> struct Arg<double> {
    double v;
    bool load(PyObject* o, bool) {
        if (!PyFloat_CheckExact(o)) return false;
        v = PyFloat_AS_DOUBLE(o);
        return true;
    }
    double get() { return v; }
    void written() {}
};
template <> struct Arg<bool> {
    bool v;
    bool load(PyObject* o, bool) {
        v = o == Py_True;
        return v || o == Py_False;
    }
    bool get() { return v; }
    void written() {}
};

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap(const std::vector<Tensor>& ts) {
    PyObject* list = PyList_New(static_cast<Py_ssize_t>(ts.size()));
    for (size_t i = 0; list && i < ts.size(); ++i) PyList_SET_ITEM(list, static_cast<Py_ssize_t>(i), THPVariable_Wrap(ts[i]));
    return list;
}
template <typename... T>
PyObject* wrap(const std::tuple<T...>& ts) {
    PyObject* tuple = PyTuple_New(sizeof...(T));
    Py_ssize_t i = 0;
    if (tuple) std::apply([&](const auto&... t) { (PyTuple_SET_ITEM(tuple, i++, wrap(t)), ...); }, ts);
    return tuple;
}

template <typename R, typename... A, size_t... I>
PyObject* call_direct(R (*function)(A...), PyObject* const* args, std::index_sequence<I...>) {
    const bool grad = at::GradMode::is_enabled();
    std::tuple<Arg<A>...> loaded;
    if (!(std::get<I>(loaded).load(args[I], grad) && ...)) Py_RETURN_NOTIMPLEMENTED;
    if constexpr (std::is_void_v<R>) {
        {
            pybind11::gil_scoped_release no_gil;
            function(std::get<I>(loaded).get()...);
        }
        (std::get<I>(loaded).written(), ...);
        Py_RETURN_NONE;
    } else {
        std::optional<R> result;
        {
            pybind11::gil_scoped_release no_gil;
            result.emplace(function(std::get<I>(loaded).get()...));
        }
        (std::get<I>(loaded).written(), ...);
        return wrap(*result);
    }
}
template <typename R, typename... A>
PyObject* call_checked(R (*function)(A...), PyObject* const* args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A)) || !nothing_interposed()) Py_RETURN_NOTIMPLEMENTED;
    return call_direct(function, args, std::index_sequence_for<A...>{});
}
template <auto kFunction>
PyObject* direct(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    return call_checked(kFunction, args, n);
    END_HANDLE_TH_ERRORS
}

// The operators that passes without a captured graph call: a position operator by operator, the single-precision step
// and the whole-sequence passes.  The 16-bit step is replayed from a graph, where a call costs the host nothing; the
// operators that only it uses go through the dispatcher.
#define METHOD(name) \
    {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&direct<&name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {METHOD(relation_select_packed), METHOD(relation_select_packed_rows), METHOD(relation_select_packed_prefill),
                          METHOD(relation_select_multi_prefill_scores), METHOD(router_cache_update), METHOD(sparse_cache_append),
                          METHOD(sequence_state), METHOD(relation_hidden_cached), METHOD(relation_hidden_cached_out),
                          METHOD(relation_hidden_cache_update), METHOD(relation_hidden_cache_update_out),
                          METHOD(relation_norm_reduce), METHOD(relation_norm_reduce_residual_norm), METHOD(relation_mlp_rows),
                          METHOD(packed_projection), METHOD(layer_norm_cast), METHOD(decode_embed_norm), METHOD(few_rows_projection),
                          METHOD(few_rows_projection_pair), METHOD(single_precision_front), METHOD(single_precision_layer),
                          METHOD(single_precision_heads), METHOD(prefill_state), METHOD(prefill_layer),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "librelation_lm_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_librelation_lm_torch() { return PyModule_Create(&kModule); }

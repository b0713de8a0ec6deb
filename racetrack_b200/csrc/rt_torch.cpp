// Tensor-level entry points: argument checks, output allocation and the call into the C ABI
// (include/rt_b200.h) of the ops that racetrack_b200/ops.py and moe.py document. A prefill hides the
// host behind its kernels; a decode step or a single-token MoE layer has kernels of 2 - 10 us, and
// checks, allocations, stream look-up and ctypes conversion in Python took 20 - 36 us a call.
//
// The module links against torch only. The kernel library's functions arrive as addresses
// (bind()), so whatever library racetrack_b200/_lib.py has loaded is the one that runs.
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <optional>
#include <string>

#include "../../include/rt_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

#define RT_TABLE(X)                                                                               \
    X(rt_last_error) X(rt_residual_norm) X(rt_rms_norm) X(rt_norm_rope_into) X(rt_rope) X(rt_swiglu)   \
    X(rt_act_quant_fp8) X(rt_swiglu_quant_fp8) X(rt_absmax) X(rt_swiglu_absmax_rows)              \
    X(rt_nvfp4_quant) X(rt_moe_route) X(rt_moe_permute_workspace_bytes) X(rt_moe_permute)         \
    X(rt_moe_tile_map) X(rt_moe_plan) X(rt_absmax_onto) X(rt_swiglu_absmax_rows_onto) X(rt_moe_gather_nvfp4) X(rt_moe_quant_nvfp4) X(rt_moe_combine)             \
    X(rt_gemm_bf16) X(rt_gemm_bf16_splitk_splits) X(rt_gemm_bf16_splitk) X(rt_gemm_bf16_batched)  \
    X(rt_gemm_fp8) X(rt_gemm_nvfp4_grouped) X(rt_index_prep_into) X(rt_index_head_weights) X(rt_fp8_index_batched)              \
    X(rt_index_topk) X(rt_mla_sparse_decode_splits) X(rt_mla_sparse_decode)

#define RT_POINTER(name) decltype(&::name) p_##name = nullptr;
RT_TABLE(RT_POINTER)
#undef RT_POINTER

void bind(const py::dict& addresses) {
#define RT_BIND(name) \
    p_##name = reinterpret_cast<decltype(&::name)>(addresses[#name].cast<uintptr_t>());
    RT_TABLE(RT_BIND)
#undef RT_BIND
}

[[noreturn]] void fail(const std::string& message) { throw std::runtime_error(message); }

void check(int status, const char* what) {
    if (status == 0) return;
    const char* msg = p_rt_last_error();
    fail(std::string(what) + " failed with status " + std::to_string(status) + ": " + (msg ? msg : ""));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void require_cuda(std::initializer_list<const Tensor*> tensors) {
    for (const Tensor* t : tensors)
        if (!t->is_cuda()) fail("racetrack_b200 ops need CUDA tensors (there is no CPU path)");
}

void require_bf16(const char* name, const Tensor& t) {
    if (t.scalar_type() != at::kBFloat16)
        fail(std::string(name) + ": expected a bfloat16 tensor, got torch." +
             std::string(c10::toString(t.scalar_type())));
}

int weight_tag(const Tensor& w) {
    if (w.scalar_type() == at::kBFloat16) return RT_BF16;
    if (w.scalar_type() == at::kFloat) return RT_F32;
    fail("norm weight must be bfloat16 or float32, got torch." + std::string(c10::toString(w.scalar_type())));
}

bool aligned16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
    return at::empty(sizes, like.options().dtype(type).layout(at::kStrided).requires_grad(false));
}

std::vector<int64_t> with_last(const Tensor& x, int64_t last) {
    std::vector<int64_t> shape = x.sizes().vec();
    shape.back() = last;
    return shape;
}

const void* ptr(const OptTensor& t) { return t ? t->data_ptr() : nullptr; }
template <typename T>
T* data(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <typename T>
T* data(const OptTensor& t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

// 2-D [rows, cols] view whose row stride the kernels can take as is: column slices of a wider
// matrix pass through, anything whose last dimension is not unit-stride or whose rows are not
// 16-byte aligned is copied.
Tensor rows_view(Tensor x) {
    const int64_t cols = x.size(-1);
    if (x.dim() == 1) x = x.unsqueeze(0);
    if (x.dim() > 2) x = x.reshape({-1, cols});
    if (x.stride(-1) != 1 || x.stride(0) % 8 != 0 || !aligned16(x)) x = x.contiguous();
    return x;
}

bool same_shape(const Tensor& t, at::IntArrayRef sizes) { return t.sizes().equals(sizes); }

// ---- norms and rotary embedding ---------------------------------------------------------------

std::tuple<Tensor, Tensor> residual_norm(const Tensor& update, const Tensor& residual, const Tensor& weight,
                                         double eps) {
    require_cuda({&update, &residual, &weight});
    require_bf16("fused_residual_norm", update);
    require_bf16("fused_residual_norm", residual);
    if (!same_shape(update, residual.sizes())) fail("fused_residual_norm: update and residual shapes differ");
    const int64_t cols = update.size(-1);
    if (weight.numel() != cols) fail("fused_residual_norm: weight length does not match the last dimension");
    const Tensor u2 = rows_view(update), r2 = rows_view(residual), w = weight.contiguous();
    Tensor normed = empty(update.sizes(), at::kBFloat16, update);
    Tensor hidden = empty(update.sizes(), at::kBFloat16, update);
    check(p_rt_residual_norm(u2.data_ptr(), r2.data_ptr(), w.data_ptr(), weight_tag(w), normed.data_ptr(),
                             hidden.data_ptr(), u2.size(0), cols, u2.stride(0), r2.stride(0),
                             static_cast<float>(eps), RT_BF16, stream()),
          "rt_residual_norm");
    return {normed, hidden};
}

Tensor rms_norm(const Tensor& x, const Tensor& weight, double eps) {
    require_cuda({&x, &weight});
    require_bf16("fused_rms_norm", x);
    const int64_t cols = x.size(-1);
    const Tensor x2 = rows_view(x), w = weight.contiguous();
    Tensor out = empty(x.sizes(), at::kBFloat16, x);
    check(p_rt_rms_norm(x2.data_ptr(), w.data_ptr(), weight_tag(w), out.data_ptr(), x2.size(0), cols,
                        x2.stride(0), cols, static_cast<float>(eps), RT_BF16, stream()),
          "rt_rms_norm");
    return out;
}

// [rows, half, 2] fp32 view of a complex64 freqs_cis tensor (no copy when contiguous)
Tensor freqs_table(const Tensor& freqs_cis, int64_t half) {
    if (!freqs_cis.is_complex()) fail("freqs_cis must be a complex tensor");
    Tensor table = at::view_as_real(freqs_cis.reshape({-1, half}).contiguous());
    return table.scalar_type() == at::kFloat ? table : table.to(at::kFloat);
}

// Whether `out` can take [rows, cols] of `type` rows in place (a slice of a cache on x's device).
bool row_slots(const Tensor& out, const Tensor& x, int64_t rows, int64_t cols, at::ScalarType type, int64_t align) {
    return out.device() == x.device() && out.scalar_type() == type && out.dim() == 2 && same_shape(out, {rows, cols}) &&
           out.stride(1) == 1 && (rows <= 1 || out.stride(0) >= cols) &&
           out.stride(0) * out.element_size() % align == 0 &&
           reinterpret_cast<uintptr_t>(out.data_ptr()) % align == 0;
}

// Python hands these on as they came: a None in the wrong place is refused, not dereferenced.
void require_one_rotation(const char* who, const OptTensor& positions, const OptTensor& inv_freq,
                          const OptTensor& freqs_cis) {
    if (positions ? !inv_freq : !freqs_cis) fail(std::string(who) + ": positions or freqs_cis is missing");
}
void require_pair(const char* who, const OptTensor& first, const OptTensor& second) {
    if (first.has_value() != second.has_value()) fail(std::string(who) + ": out must be a pair of tensors");
}

// positions + inverse frequencies (half-split pairs), or a complex table (interleaved pairs)
std::tuple<Tensor, Tensor, Tensor> norm_rope(const Tensor& q_c, const Tensor& q_weight, const Tensor& kv_c,
                                             const Tensor& kv_weight, const Tensor& k_pe,
                                             const OptTensor& positions, const OptTensor& inv_freq,
                                             const OptTensor& freqs_cis, double eps, const OptTensor& kv_into,
                                             const OptTensor& k_into) {
    require_one_rotation("fused_norm_rope", positions, inv_freq, freqs_cis);
    Tensor pos, table;
    int mode = RT_ROPE_INTERLEAVED;
    int64_t table_rows = 0;
    if (positions) {
        pos = positions->reshape(-1).to(at::kLong).contiguous();
        table = *inv_freq;
        mode = RT_ROPE_HALF;
    } else {
        table = freqs_table(*freqs_cis, k_pe.size(-1) / 2);
        table_rows = table.size(0);
    }
    require_cuda({&q_c, &kv_c, &k_pe, &q_weight, &kv_weight});
    require_bf16("fused_norm_rope q_c", q_c);
    require_bf16("fused_norm_rope kv_c", kv_c);
    require_bf16("fused_norm_rope k_pe", k_pe);
    const Tensor q2 = rows_view(q_c), kv2 = rows_view(kv_c);
    Tensor k2 = k_pe.dim() == 2 ? k_pe : k_pe.reshape({-1, k_pe.size(-1)});
    if (k2.stride(-1) != 1) k2 = k2.contiguous();
    const int64_t tokens = q2.size(0);
    if (kv2.size(0) != tokens || k2.size(0) != tokens)
        fail("fused_norm_rope: q_c, kv_c and k_pe disagree on the token count");
    const Tensor qw = q_weight.contiguous();
    Tensor kvw = kv_weight.contiguous();
    if (qw.scalar_type() != kvw.scalar_type()) kvw = kvw.to(qw.scalar_type());
    Tensor q_out = empty(q_c.sizes(), at::kBFloat16, q_c);
    // into the caller's rows where they can be written as they are, else a tensor and a copy
    const bool into = kv_into && k_into && row_slots(*kv_into, q_c, tokens, kv2.size(1), at::kBFloat16, 16) &&
                      row_slots(*k_into, q_c, tokens, k2.size(1), at::kBFloat16, 2);
    Tensor kv_out = into ? *kv_into : empty(kv_c.sizes(), at::kBFloat16, kv_c);
    Tensor k_out = into ? *k_into : empty(k_pe.sizes(), at::kBFloat16, k_pe);
    check(p_rt_norm_rope_into(q2.data_ptr(), qw.data_ptr(), kv2.data_ptr(), kvw.data_ptr(), weight_tag(qw),
                         k2.data_ptr(), pos.defined() ? data<int64_t>(pos) : nullptr, data<float>(table),
                         table_rows, q_out.data_ptr(), kv_out.data_ptr(), k_out.data_ptr(), tokens, q2.size(1),
                         kv2.size(1), k2.size(1), q2.stride(0), kv2.stride(0), k2.stride(0),
                         into ? kv_out.stride(0) : kv2.size(1), into ? k_out.stride(0) : k2.size(1),
                         static_cast<float>(eps), mode, RT_BF16, stream()),
          "rt_norm_rope");
    if (into) {
        kv_out.unsafeGetTensorImpl()->bump_version();
        k_out.unsafeGetTensorImpl()->bump_version();
    } else if (kv_into && k_into) {
        kv_into->copy_(kv_out);
        k_into->copy_(k_out);
    }
    return {q_out, kv_out, k_out};
}

Tensor rope(const Tensor& x, const OptTensor& positions, const OptTensor& inv_freq, const OptTensor& freqs_cis,
            bool inplace) {
    require_one_rotation("fused_rope", positions, inv_freq, freqs_cis);
    Tensor pos, table;
    int mode = RT_ROPE_INTERLEAVED;
    int64_t table_rows = 0;
    if (positions) {
        pos = positions->reshape(-1).to(at::kLong).contiguous();
        table = *inv_freq;
        mode = RT_ROPE_HALF;
    } else {
        table = freqs_table(*freqs_cis, x.size(-1) / 2);
        table_rows = table.size(0);
    }
    require_cuda({&x});
    require_bf16("fused_rope", x);
    if (x.dim() < 2) fail("fused_rope: expected [..., heads, rope_dim]");
    const int64_t d = x.size(-1), heads = x.size(-2);
    Tensor x3 = x.dim() != 3 ? x.reshape({-1, heads, d}) : x;
    if (x3.stride(2) != 1 || x3.stride(0) % 8 != 0 || x3.stride(1) % 8 != 0 || !aligned16(x3)) {
        if (inplace) fail("fused_rope: in-place rotation needs a 16-byte aligned strided view");
        x3 = x3.contiguous();
    }
    Tensor out3 = inplace ? x3 : empty({x3.size(0), heads, d}, at::kBFloat16, x);
    check(p_rt_rope(x3.data_ptr(), pos.defined() ? data<int64_t>(pos) : nullptr, data<float>(table), table_rows,
                    out3.data_ptr(), x3.size(0), heads, d, x3.stride(0), x3.stride(1), out3.stride(0),
                    out3.stride(1), mode, RT_BF16, stream()),
          "rt_rope");
    return inplace ? x : out3.view(x.sizes());
}

// ---- SwiGLU and quantisers ----------------------------------------------------------------------

std::pair<Tensor, Tensor> gate_up(const Tensor& gate, const Tensor& up, const char* who) {
    require_cuda({&gate, &up});
    require_bf16(who, gate);
    require_bf16(who, up);
    if (!same_shape(gate, up.sizes())) fail(std::string(who) + ": gate and up shapes differ");
    return {rows_view(gate), rows_view(up)};
}

Tensor swiglu(const Tensor& gate, const Tensor& up) {
    const auto [g2, u2] = gate_up(gate, up, "fused_swiglu");
    Tensor out = empty(gate.sizes(), at::kBFloat16, gate);
    check(p_rt_swiglu(g2.data_ptr(), u2.data_ptr(), out.data_ptr(), g2.size(0), g2.size(1), g2.stride(0),
                      u2.stride(0), RT_BF16, stream()),
          "rt_swiglu");
    return out;
}

std::tuple<Tensor, Tensor> act_quant(const Tensor& x, const OptTensor& out_codes, const OptTensor& out_scales) {
    require_pair("fused_act_quant", out_codes, out_scales);
    require_cuda({&x});
    require_bf16("fused_act_quant", x);
    const int64_t n = x.size(-1);
    if (n % 128 != 0)
        fail("fused_act_quant: last dim (" + std::to_string(n) + ") must be a multiple of 128");
    const Tensor x2 = rows_view(x);
    Tensor codes, scales;
    if (out_codes) {
        codes = *out_codes;
        scales = *out_scales;
        if (codes.element_size() != 1 || scales.scalar_type() != at::kFloat || !codes.is_contiguous() ||
            !scales.is_contiguous() || !same_shape(codes, x.sizes()) || !same_shape(scales, with_last(x, n / 128)))
            fail("fused_act_quant: out must be contiguous (1-byte codes [..., N], fp32 scales [..., N/128])");
    } else {
        codes = empty(x.sizes(), at::kFloat8_e4m3fn, x);
        scales = empty(with_last(x, n / 128), at::kFloat, x);
    }
    check(p_rt_act_quant_fp8(x2.data_ptr(), codes.data_ptr(), data<float>(scales), x2.size(0), n, x2.stride(0),
                             RT_BF16, stream()),
          "rt_act_quant_fp8");
    return {codes, scales};
}

std::tuple<Tensor, Tensor> swiglu_quant(const Tensor& gate, const Tensor& up) {
    const auto [g2, u2] = gate_up(gate, up, "fused_swiglu_quant");
    const int64_t n = gate.size(-1);
    if (n % 128 != 0)
        fail("fused_swiglu_quant: last dim (" + std::to_string(n) + ") must be a multiple of 128");
    Tensor codes = empty(gate.sizes(), at::kFloat8_e4m3fn, gate);
    Tensor scales = empty(with_last(gate, n / 128), at::kFloat, gate);
    check(p_rt_swiglu_quant_fp8(g2.data_ptr(), u2.data_ptr(), codes.data_ptr(), data<float>(scales), g2.size(0),
                                n, g2.stride(0), u2.stride(0), RT_BF16, stream()),
          "rt_swiglu_quant_fp8");
    return {codes, scales};
}

Tensor tensor_absmax(const Tensor& x, const OptTensor& up) {
    require_cuda({&x});
    require_bf16("tensor_absmax", x);
    if (x.size(-1) % 16 != 0) fail("tensor_absmax: last dim must be a multiple of 16");
    const Tensor x2 = rows_view(x);
    OptTensor u2;
    if (up) u2 = rows_view(*up);
    Tensor out = empty({1}, at::kFloat, x);
    check(p_rt_absmax(x2.data_ptr(), ptr(u2), data<float>(out), x2.size(0), x2.size(1), x2.stride(0),
                      u2 ? u2->stride(0) : 0, RT_BF16, stream()),
          "rt_absmax");
    return out;
}

std::tuple<Tensor, Tensor> swiglu_absmax(const Tensor& gate, const Tensor& up, const OptTensor& begin,
                                         const OptTensor& end) {
    Tensor h = empty(gate.sizes(), at::kBFloat16, gate), out = empty({1}, at::kFloat, gate);
    check(p_rt_swiglu_absmax_rows(gate.data_ptr(), up.data_ptr(), h.data_ptr(), data<float>(out), gate.size(0),
                                  gate.size(1), gate.stride(0), up.stride(0), h.stride(0), data<int32_t>(begin),
                                  data<int32_t>(end), RT_BF16, stream()),
          "rt_swiglu_absmax_rows");
    return {h, out};
}

int64_t sf_tiled_bytes(int64_t rows, int64_t cols) { return ((rows + 127) / 128) * ((cols / 16 + 3) / 4) * 512; }

std::tuple<Tensor, Tensor, Tensor> nvfp4_quant(const Tensor& x, const OptTensor& up, const OptTensor& amax_in,
                                               bool tiled, const OptTensor& out_codes, const OptTensor& out_sf) {
    require_pair("fused_nvfp4_quant", out_codes, out_sf);
    require_cuda({&x});
    require_bf16("fused_nvfp4_quant", x);
    const int64_t n = x.size(-1);
    if (n % 16 != 0)
        fail("fused_nvfp4_quant: last dim (" + std::to_string(n) + ") must be a multiple of 16");
    Tensor x2;
    OptTensor u2;
    if (up) {
        auto [g, u] = gate_up(x, *up, "fused_nvfp4_quant");
        x2 = g;
        u2 = u;
    } else {
        x2 = rows_view(x);
    }
    Tensor amax;
    if (amax_in) {
        amax = *amax_in;
    } else if (up && x2.size(0) > 0) {
        // one evaluation of SwiGLU: the abs-max pass writes its bf16 result and the quantiser reads
        // that (4 + 2 + 2 + 0.56 bytes an element, as many as two passes over gate and up move, at
        // half the instructions; 4096 x 18432 on one B200: 120 us against 161)
        std::tie(x2, amax) = swiglu_absmax(x2, *u2, std::nullopt, std::nullopt);
        u2.reset();
    } else {
        amax = tensor_absmax(x, up);
    }
    const int64_t rows = x2.size(0);
    Tensor codes, sf;
    const std::vector<int64_t> sf_shape =
        tiled ? std::vector<int64_t>{sf_tiled_bytes(rows, n)} : with_last(x, n / 16);
    if (out_codes) {
        codes = *out_codes;
        sf = *out_sf;
        if (codes.scalar_type() != at::kByte || sf.scalar_type() != at::kByte || !codes.is_contiguous() ||
            !sf.is_contiguous() || !same_shape(codes, with_last(x, n / 2)) || !same_shape(sf, sf_shape))
            fail("fused_nvfp4_quant: out must be contiguous uint8 (codes [..., N/2], scales)");
    } else {
        codes = empty(with_last(x, n / 2), at::kByte, x);
        sf = empty(sf_shape, at::kByte, x);
    }
    Tensor gs = empty({1}, at::kFloat, x);
    check(p_rt_nvfp4_quant(x2.data_ptr(), ptr(u2), data<float>(amax), codes.data_ptr(), sf.data_ptr(),
                           data<float>(gs), rows, n, x2.stride(0), u2 ? u2->stride(0) : 0,
                           tiled ? RT_SF_TILED128x4 : RT_SF_ROWMAJOR, RT_BF16, stream()),
          "rt_nvfp4_quant");
    return {codes, sf.view(at::kFloat8_e4m3fn), gs};
}

// ---- tensor-core GEMMs ---------------------------------------------------------------------------

Tensor out_buffer(const OptTensor& out, at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
    if (!out) return empty(shape, type, like);
    if (!same_shape(*out, shape) || out->scalar_type() != type || !out->is_contiguous()) {
        std::string text;
        for (int64_t s : shape) text += std::to_string(s) + ", ";
        fail("out must be a contiguous torch." + std::string(c10::toString(type)) + " tensor of shape (" + text + ")");
    }
    return *out;
}

Tensor linear_bf16(const Tensor& x, const Tensor& weight, bool f32_out, const OptTensor& out_in,
                   int64_t splitk_max_rows) {
    require_cuda({&x, &weight});
    require_bf16("linear_bf16 x", x);
    require_bf16("linear_bf16 weight", weight);
    const int64_t k = x.size(-1);
    if (weight.dim() != 2 || weight.size(1) != k) fail("linear_bf16: weight must be [N, K] with K matching x");
    const Tensor x2 = rows_view(x);
    const Tensor w =
        weight.stride(1) == 1 && weight.stride(0) % 8 == 0 && aligned16(weight) ? weight : weight.contiguous();
    const int64_t n = w.size(0), rows = x2.size(0);
    const at::ScalarType type = f32_out ? at::kFloat : at::kBFloat16;
    const int tag = f32_out ? RT_F32 : RT_BF16;
    // a few decode tokens have too few output tiles to occupy the GPU: the library says, by the
    // weight's shape, into how many ranges to cut K
    const int64_t splits = rows > 0 && rows <= splitk_max_rows ? p_rt_gemm_bf16_splitk_splits(rows, n, k) : 1;
    if (splits > 1) {
        // partial products per K range, then their sum in a fixed order: bit-reproducible, and
        // identical on every rank that forms the same replicated projection
        Tensor part = empty({splits, rows, n}, at::kFloat, x);
        Tensor out = out_buffer(out_in, with_last(x, n), type, x);
        check(p_rt_gemm_bf16_splitk(x2.data_ptr(), w.data_ptr(), data<float>(part), out.data_ptr(), rows, n, k,
                                    x2.stride(0), w.stride(0), n, n, splits, tag, stream()),
              "rt_gemm_bf16_splitk");
        return out;
    }
    Tensor out = out_buffer(out_in, with_last(x, n), type, x);
    check(p_rt_gemm_bf16(x2.data_ptr(), w.data_ptr(), out.data_ptr(), rows, n, k, x2.stride(0), w.stride(0), n, tag,
                         stream()),
          "rt_gemm_bf16");
    return out;
}

Tensor linear_bf16_batched(Tensor x, Tensor weight) {
    require_cuda({&x, &weight});
    require_bf16("linear_bf16_batched x", x);
    require_bf16("linear_bf16_batched weight", weight);
    if (x.dim() != 3 || weight.dim() != 3 || weight.size(0) != x.size(1) || weight.size(2) != x.size(2))
        fail("linear_bf16_batched: expected x [T, H, K] and weight [H, N, K]");
    if (x.stride(2) != 1 || x.stride(0) % 8 || x.stride(1) % 8 || !aligned16(x)) x = x.contiguous();
    if (weight.stride(2) != 1 || weight.stride(0) % 8 || weight.stride(1) % 8 || !aligned16(weight))
        weight = weight.contiguous();
    const int64_t tokens = x.size(0), heads = x.size(1), k = x.size(2), n = weight.size(1);
    Tensor out = empty({tokens, heads, n}, at::kBFloat16, x);
    check(p_rt_gemm_bf16_batched(x.data_ptr(), weight.data_ptr(), out.data_ptr(), heads, tokens, n, k, x.stride(0),
                                 x.stride(1), weight.stride(1), weight.stride(0), out.stride(0), out.stride(1),
                                 stream()),
          "rt_gemm_bf16_batched");
    return out;
}

Tensor linear_fp8(const Tensor& x_codes, const Tensor& x_scales, const Tensor& w_codes, const Tensor& w_scales,
                  const OptTensor& out_in) {
    require_cuda({&x_codes, &x_scales, &w_codes, &w_scales});
    const int64_t k = x_codes.size(-1), n = w_codes.size(0);
    if (w_codes.size(1) != k || x_codes.scalar_type() != at::kFloat8_e4m3fn ||
        w_codes.scalar_type() != at::kFloat8_e4m3fn)
        fail("linear_fp8: expected e4m3fn codes with matching K");
    const Tensor xc = x_codes.reshape({-1, k}), xs = x_scales.reshape({-1, k / 128});
    if (!xc.is_contiguous() || !xs.is_contiguous() || !w_codes.is_contiguous() || !w_scales.is_contiguous())
        fail("linear_fp8: operands must be contiguous");
    if (xs.scalar_type() != at::kFloat || w_scales.scalar_type() != at::kFloat ||
        !same_shape(w_scales, {(n + 127) / 128, k / 128}))
        fail("linear_fp8: scales must be fp32 [M, K/128] and [ceil(N/128), K/128]");
    Tensor out = out_buffer(out_in, with_last(x_codes, n), at::kBFloat16, x_codes);
    check(p_rt_gemm_fp8(xc.data_ptr(), data<float>(xs), w_codes.data_ptr(), data<float>(w_scales), out.data_ptr(),
                        xc.size(0), n, k, k, k, n, stream()),
          "rt_gemm_fp8");
    return out;
}

Tensor gemm_nvfp4_grouped(const Tensor& a_codes, const Tensor& a_sf, const Tensor& a_gs, const Tensor& b_codes,
                          const Tensor& b_sf, const Tensor& b_gs, const Tensor& tile_map, const Tensor& tile_count,
                          int64_t n, int64_t groups, const OptTensor& out_in) {
    require_cuda({&a_codes, &a_sf, &a_gs, &b_codes, &b_sf, &b_gs, &tile_map, &tile_count});
    if (a_codes.dim() != 2) fail("gemm_nvfp4_grouped: a_codes must be [rows, K/2]");
    const int64_t rows = a_codes.size(0), kh = a_codes.size(1);
    if (!same_shape(b_codes, {groups * n, kh})) fail("gemm_nvfp4_grouped: b_codes must be [groups * n, K/2]");
    if (!a_codes.is_contiguous() || !b_codes.is_contiguous())
        fail("gemm_nvfp4_grouped: code tensors must be contiguous");
    Tensor out = out_in ? *out_in : empty({rows, n}, at::kBFloat16, a_codes);
    check(p_rt_gemm_nvfp4_grouped(a_codes.data_ptr(), a_sf.data_ptr(), data<float>(a_gs), b_codes.data_ptr(),
                                  b_sf.data_ptr(), data<float>(b_gs), out.data_ptr(), data<int32_t>(tile_map),
                                  data<int32_t>(tile_count), tile_map.size(0) / 2, rows, groups, n, 2 * kh,
                                  out.stride(0), stream()),
          "rt_gemm_nvfp4_grouped");
    return out;
}

// ---- mixture of experts --------------------------------------------------------------------------

std::tuple<Tensor, Tensor> moe_route(Tensor logits, OptTensor bias, int64_t n_groups, int64_t topk_groups,
                                     int64_t topk, double route_scale, int score_func, const OptTensor& out_weights,
                                     const OptTensor& out_indices) {
    require_pair("fused_moe_route", out_weights, out_indices);
    require_cuda({&logits});
    if (logits.scalar_type() != at::kFloat || logits.dim() != 2)
        fail("fused_moe_route: logits must be a 2-D float32 tensor");
    if (logits.stride(1) != 1) logits = logits.contiguous();
    if (bias) bias = bias->to(at::kFloat).contiguous();
    const int64_t tokens = logits.size(0), n_experts = logits.size(1);
    Tensor weights, indices;
    if (out_weights) {
        weights = *out_weights;
        indices = *out_indices;
        if (weights.scalar_type() != at::kFloat || indices.scalar_type() != at::kLong || !weights.is_contiguous() ||
            !indices.is_contiguous() || !same_shape(weights, {tokens, topk}) || !same_shape(indices, {tokens, topk}))
            fail("fused_moe_route: out must be contiguous (fp32 [T, topk], int64 [T, topk])");
    } else {
        weights = empty({tokens, topk}, at::kFloat, logits);
        indices = empty({tokens, topk}, at::kLong, logits);
    }
    check(p_rt_moe_route(data<float>(logits), data<float>(bias), data<float>(weights), data<int64_t>(indices), tokens,
                         n_experts, logits.stride(0), n_groups, topk_groups, topk, static_cast<float>(route_scale),
                         score_func, stream()),
          "rt_moe_route");
    return {weights, indices};
}

std::tuple<Tensor, Tensor, Tensor> moe_permute(Tensor indices, int64_t n_experts) {
    require_cuda({&indices});
    if (indices.scalar_type() != at::kLong || indices.dim() != 2)
        fail("fused_moe_permute: indices must be a 2-D int64 tensor");
    indices = indices.contiguous();
    const int64_t tokens = indices.size(0), topk = indices.size(1);
    const int64_t ws = p_rt_moe_permute_workspace_bytes(tokens, topk, n_experts);
    Tensor workspace = empty({std::max<int64_t>(ws, 4)}, at::kByte, indices);
    Tensor offsets = empty({n_experts + 1}, at::kInt, indices);
    Tensor sorted_pairs = empty({tokens * topk}, at::kInt, indices);
    Tensor pair_pos = empty({tokens * topk}, at::kInt, indices);
    check(p_rt_moe_permute(data<int64_t>(indices), data<int32_t>(offsets), data<int32_t>(sorted_pairs),
                           data<int32_t>(pair_pos), workspace.data_ptr(), tokens, topk, n_experts, stream()),
          "rt_moe_permute");
    return {offsets, sorted_pairs, pair_pos};
}

std::tuple<Tensor, Tensor, Tensor> moe_tile_map(const Tensor& offsets, int64_t g_begin, int64_t g_end,
                                                int64_t max_tiles) {
    require_cuda({&offsets});
    if (offsets.scalar_type() != at::kInt) fail("moe_tile_map: offsets must be int32");
    Tensor tile_map = empty({2 * max_tiles, 4}, at::kInt, offsets);
    Tensor tile_base = empty({g_end - g_begin + 1}, at::kInt, offsets);
    Tensor tile_count = empty({2}, at::kInt, offsets);
    check(p_rt_moe_tile_map(data<int32_t>(offsets), g_begin, g_end, data<int32_t>(tile_map), data<int32_t>(tile_base),
                            data<int32_t>(tile_count), max_tiles, stream()),
          "rt_moe_tile_map");
    return {tile_map, tile_base, tile_count};
}

std::tuple<Tensor, Tensor> moe_gather_nvfp4(const Tensor& codes, const Tensor& sf, const Tensor& sorted_pairs,
                                            int64_t topk, const Tensor& tile_map, const Tensor& tile_count,
                                            int64_t total_rows) {
    const int64_t cols = codes.size(1) * 2, max_tiles = tile_map.size(0) / 2;
    Tensor out = empty({total_rows, cols / 2}, at::kByte, codes);
    Tensor sf_out = empty({max_tiles * (cols / 64) * 512}, at::kByte, codes);
    check(p_rt_moe_gather_nvfp4(codes.data_ptr(), sf.data_ptr(), data<int32_t>(sorted_pairs), topk, out.data_ptr(),
                                sf_out.data_ptr(), data<int32_t>(tile_map), data<int32_t>(tile_count), max_tiles,
                                cols, stream()),
          "rt_moe_gather_nvfp4");
    return {out, sf_out};
}

std::tuple<Tensor, Tensor, Tensor> moe_quant_nvfp4(const Tensor& x, const Tensor& tile_map, const Tensor& tile_count,
                                                   int64_t total_rows, const Tensor& amax,
                                                   const OptTensor& sorted_pairs, int64_t topk, const OptTensor& up) {
    const int64_t cols = x.size(-1), max_tiles = tile_map.size(0) / 2;
    Tensor codes = empty({total_rows, cols / 2}, at::kByte, x);
    Tensor sf = empty({max_tiles * (cols / 64) * 512}, at::kByte, x);
    Tensor gs = empty({1}, at::kFloat, x);
    check(p_rt_moe_quant_nvfp4(x.data_ptr(), ptr(up), data<int32_t>(sorted_pairs), topk, data<float>(amax),
                               codes.data_ptr(), sf.data_ptr(), data<float>(gs), data<int32_t>(tile_map),
                               data<int32_t>(tile_count), max_tiles, cols, x.stride(0), up ? up->stride(0) : 0,
                               RT_BF16, stream()),
          "rt_moe_quant_nvfp4");
    return {codes, sf, gs};
}

Tensor moe_combine(Tensor expert_out, const Tensor& pair_pos, Tensor weights, OptTensor shared, int64_t pos_begin,
                   std::optional<int64_t> pos_end, const OptTensor& window_begin, const OptTensor& window_end,
                   bool f32_out, const OptTensor& out) {
    require_cuda({&expert_out, &pair_pos, &weights});
    require_bf16("fused_moe_combine", expert_out);
    const int64_t tokens = weights.size(0), topk = weights.size(1), cols = expert_out.size(-1);
    if (pair_pos.numel() < tokens * topk) fail("fused_moe_combine: pair_pos must have a position for every weight");
    expert_out = expert_out.contiguous();
    weights = weights.to(at::kFloat).contiguous();
    if (shared) {
        require_bf16("fused_moe_combine", *shared);
        shared = shared->reshape({tokens, cols}).contiguous();
    }
    Tensor y = out_buffer(out, {tokens, cols}, f32_out ? at::kFloat : at::kBFloat16, expert_out);
    check(p_rt_moe_combine(expert_out.data_ptr(), data<int32_t>(pair_pos), data<float>(weights), ptr(shared),
                           y.data_ptr(), tokens, topk, cols, pos_begin, pos_end.value_or(tokens * topk),
                           data<int32_t>(window_begin), data<int32_t>(window_end), f32_out ? RT_F32 : RT_BF16,
                           stream()),
          "rt_moe_combine");
    return y;
}

// The whole routed-expert MLP (racetrack_b200/moe.py, fused_moe_experts). Returns y and, for
// stage-wise checks, (offsets, sorted_pairs, pair_pos, x_gs, x_amax, gate_up, h, h_amax, expert_out).
using Experts = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, OptTensor, Tensor, Tensor, Tensor, Tensor>;
Experts moe_experts(const OptTensor& x, const Tensor& weights, const Tensor& indices, const Tensor& w13_codes,
                      const Tensor& w13_sf, const Tensor& w13_gs, const Tensor& w2_codes, const Tensor& w2_sf,
                      const Tensor& w2_gs, int64_t count, int64_t inter, int64_t n_experts, int64_t expert_begin,
                      const OptTensor& shared, bool f32_out, const OptTensor& q_codes, const OptTensor& q_sf,
                      const OptTensor& q_gs, const OptTensor& out, const std::optional<py::function>& around_w13) {
    if (q_codes ? !(q_sf && q_gs) : !x) fail("fused_moe_experts: x or x_quant (codes, scales, global scale) is required");
    const Tensor& in = q_codes ? *q_codes : *x;
    if (in.dim() != 2) fail("fused_moe_experts: x must be [T, hidden] (x_quant codes [T, hidden / 2])");
    if (indices.scalar_type() != at::kLong || indices.dim() != 2)
        fail("fused_moe_permute: indices must be a 2-D int64 tensor");
    // the routed rows are those of indices: they name rows of x, and weights has one value for each
    const int64_t tokens = indices.size(0), topk = indices.size(1), pairs = tokens * topk;
    if (tokens > in.size(0) || weights.dim() != 2 || weights.size(0) > tokens || weights.size(1) != topk)
        fail("fused_moe_experts: x, weights and indices disagree on the token count or on topk");
    const int64_t hidden = q_codes ? in.size(1) * 2 : in.size(1);
    require_cuda({&indices, &in});
    const Tensor idx = indices.contiguous();
    const int64_t max_tiles = (pairs + 127) / 128 + count;
    Tensor workspace = empty(
        {std::max<int64_t>(p_rt_moe_permute_workspace_bytes(tokens, topk, n_experts), 4)}, at::kByte, idx);
    Tensor offsets = empty({n_experts + 1}, at::kInt, idx), sorted_pairs = empty({pairs}, at::kInt, idx);
    Tensor pair_pos = empty({pairs}, at::kInt, idx), tile_map = empty({2 * max_tiles, 4}, at::kInt, idx);
    Tensor tile_base = empty({count + 1}, at::kInt, idx), tile_count = empty({2}, at::kInt, idx);
    Tensor amax2 = empty({2}, at::kFloat, idx);           // of x and of h, zeroed by the plan
    check(p_rt_moe_plan(data<int64_t>(idx), data<int32_t>(offsets), data<int32_t>(sorted_pairs),
                        data<int32_t>(pair_pos), workspace.data_ptr(), data<int32_t>(tile_map),
                        data<int32_t>(tile_base), data<int32_t>(tile_count), data<float>(amax2), max_tiles,
                        expert_begin, expert_begin + count, tokens, topk, n_experts, stream()),
          "rt_moe_plan");
    OptTensor begin, end;
    if (count != n_experts) {
        begin = offsets.slice(0, expert_begin, expert_begin + 1);
        end = offsets.slice(0, expert_begin + count, expert_begin + count + 1);
    }
    Tensor a_codes, a_sf, x_gs;
    OptTensor x_amax;
    if (q_codes) {
        x_gs = *q_gs;
        std::tie(a_codes, a_sf) = moe_gather_nvfp4(*q_codes, *q_sf, sorted_pairs, topk, tile_map, tile_count, pairs);
    } else {
        require_bf16("tensor_absmax", *x);
        if (hidden % 16 != 0) fail("tensor_absmax: last dim must be a multiple of 16");
        const Tensor x2 = rows_view(*x);
        x_amax = amax2.slice(0, 0, 1);
        check(p_rt_absmax_onto(x2.data_ptr(), data<float>(amax2), x2.size(0), hidden, x2.stride(0), RT_BF16, stream()),
              "rt_absmax_onto");
        if (pairs <= 256) {
            // few rows: quantised straight into expert order, once per pair, instead of once per token
            // and copied; the same bits (7168 columns, top 8, one B200: 1 token 6 us against 11 in two
            // launches, 13 tokens 9 / 12; 64 tokens 17 / 14)
            std::tie(a_codes, a_sf, x_gs) =
                moe_quant_nvfp4(x2, tile_map, tile_count, pairs, *x_amax, sorted_pairs, topk, std::nullopt);
        } else {
            // every token row is quantised once, then its codes and scales are copied into expert
            // order (the bf16 rows are not read topk times)
            auto [x_codes, x_sf, gs] = nvfp4_quant(*x, std::nullopt, x_amax, false, std::nullopt, std::nullopt);
            x_gs = gs;
            std::tie(a_codes, a_sf) = moe_gather_nvfp4(x_codes, x_sf, sorted_pairs, topk, tile_map, tile_count, pairs);
        }
    }
    auto around = [&](bool begin) {
        if (!around_w13) return;
        py::gil_scoped_acquire gil;
        (*around_w13)(begin);
    };
    around(true);
    Tensor gate_up_out = gemm_nvfp4_grouped(a_codes, a_sf, x_gs, w13_codes, w13_sf, w13_gs, tile_map, tile_count,
                                            2 * inter, count, std::nullopt);
    around(false);
    // SwiGLU once: this pass writes h and finds the tensor-wide amax its quantisation needs
    const Tensor gate = gate_up_out.slice(1, 0, inter), up = gate_up_out.slice(1, inter, 2 * inter);
    Tensor h = empty({pairs, inter}, at::kBFloat16, gate_up_out), h_amax = amax2.slice(0, 1, 2);
    check(p_rt_swiglu_absmax_rows_onto(gate.data_ptr(), up.data_ptr(), h.data_ptr(), data<float>(h_amax), pairs, inter,
                                       gate.stride(0), up.stride(0), inter, data<int32_t>(begin), data<int32_t>(end),
                                       RT_BF16, stream()),
          "rt_swiglu_absmax_rows_onto");
    auto [h_codes, h_sf, h_gs] = moe_quant_nvfp4(h, tile_map, tile_count, pairs, h_amax, std::nullopt, 1, std::nullopt);
    Tensor expert_out = gemm_nvfp4_grouped(h_codes, h_sf, h_gs, w2_codes, w2_sf, w2_gs, tile_map, tile_count, hidden,
                                           count, std::nullopt);
    Tensor y = moe_combine(expert_out, pair_pos, weights, shared, 0, std::nullopt, begin, end, f32_out, out);
    return {y, offsets, sorted_pairs, pair_pos, x_gs, x_amax, gate_up_out, h, h_amax, expert_out};
}

// ---- sparse indexer and decode attention -----------------------------------------------------------

std::tuple<Tensor, Tensor, OptTensor> index_prep(const Tensor& x, const Tensor& freqs_cis, const OptTensor& positions, const OptTensor& ln_weight,
                     const OptTensor& ln_bias, double eps, bool return_rotated, const OptTensor& codes_into,
                     const OptTensor& scales_into) {
    require_cuda({&x, &freqs_cis});
    require_bf16("index_prep", x);
    if (x.dim() != 3 || x.size(-1) != 128) fail("index_prep: x must be [S, H, 128]");
    const int64_t s_len = x.size(0), heads = x.size(1), dim = x.size(2);
    Tensor x2 = x.reshape({s_len * heads, dim});
    if (x2.stride(1) != 1) x2 = x2.contiguous();
    const Tensor fr = at::view_as_real(freqs_cis).to(at::kFloat).contiguous();
    if (fr.dim() < 2 || fr.size(-2) != 32 || fr.size(-1) != 2) fail("index_prep: freqs_cis must be [table, 32] complex");
    // one key per token: into the caller's cache rows where they can be written as they are
    const bool into = codes_into && scales_into && heads == 1 &&
                      row_slots(*codes_into, x, s_len, dim, at::kFloat8_e4m3fn, 4) &&
                      scales_into->device() == x.device() &&
                      scales_into->scalar_type() == at::kFloat && scales_into->dim() == 1 &&
                      scales_into->size(0) == s_len && (s_len <= 1 || scales_into->stride(0) >= 1);
    Tensor codes = into ? *codes_into : empty({s_len, heads, dim}, at::kFloat8_e4m3fn, x);
    Tensor scales = into ? *scales_into : empty({s_len, heads}, at::kFloat, x);
    OptTensor rotated, lw, lb, pos;
    if (return_rotated) rotated = empty({s_len, heads, dim}, at::kBFloat16, x);
    if (ln_weight) lw = ln_weight->to(at::kFloat).contiguous();
    if (ln_bias) lb = ln_bias->to(at::kFloat).contiguous();
    if (positions) pos = positions->to(at::kLong).contiguous();
    check(p_rt_index_prep_into(x2.data_ptr(), data<float>(lw), data<float>(lb), data<int64_t>(pos), data<float>(fr),
                          fr.size(0), heads, codes.data_ptr(), data<float>(scales),
                          rotated ? rotated->data_ptr() : nullptr, s_len * heads, dim, 64, x2.stride(0),
                          into ? codes.stride(0) : dim, into ? scales.stride(0) : 1,
                          static_cast<float>(eps), RT_BF16, stream()),
          "rt_index_prep");
    if (into) {
        codes.unsafeGetTensorImpl()->bump_version();
        scales.unsafeGetTensorImpl()->bump_version();
    } else if (codes_into && scales_into) {
        codes_into->copy_(codes.view({s_len, heads * dim}));
        scales_into->copy_(scales.view({s_len * heads}));
    }
    return {codes, scales, rotated};
}

Tensor index_head_weights(const Tensor& both, const Tensor& q_scale, double c1, double c2) {
    require_cuda({&both, &q_scale});
    const int64_t rows = q_scale.size(0), heads = q_scale.size(1);
    if (both.scalar_type() != at::kFloat || q_scale.scalar_type() != at::kFloat || q_scale.dim() != 2 ||
        !same_shape(both, {rows, 2 * heads}) || !both.is_contiguous() || !q_scale.is_contiguous())
        fail("index_head_weights: expected contiguous fp32 [S, 2 * H] and [S, H]");
    Tensor out = empty({rows, heads}, at::kFloat, both);
    check(p_rt_index_head_weights(data<float>(both), data<float>(q_scale), data<float>(out), rows, heads,
                                  static_cast<float>(c1), static_cast<float>(c2), stream()),
          "rt_index_head_weights");
    return out;
}

Tensor fp8_index(const Tensor& q, const Tensor& weights, const Tensor& k, const Tensor& k_scale,
                 std::optional<int64_t> causal_offset) {
    require_cuda({&q, &weights, &k, &k_scale});
    if (q.scalar_type() != at::kFloat8_e4m3fn || k.scalar_type() != at::kFloat8_e4m3fn)
        fail("fp8_index: q and k must be float8_e4m3fn");
    if (q.dim() < 3 || k.dim() < 2 || q.dim() > 4 || k.dim() != q.dim() - 1 ||
        (q.dim() == 4 && k.size(0) != q.size(0)))
        fail("fp8_index: q [B, M, H, D] and k [B, N, D] must share at most one batch dim");
    const int64_t m = q.size(-3), h = q.size(-2), d = q.size(-1), n = k.size(-2);
    const bool lead = q.dim() == 4;
    const int64_t batch = lead ? q.size(0) : 1;
    const Tensor q3 = q.reshape({batch, m, h, d}).contiguous();
    Tensor k3 = k.reshape({batch, n, d});
    if (k3.stride(2) != 1 || k3.stride(1) != d || (batch > 1 && k3.stride(0) % d)) k3 = k3.contiguous();
    const Tensor w3 = weights.reshape({batch, m, h}).to(at::kFloat).contiguous();
    Tensor ks = k_scale.reshape({batch, n}).to(at::kFloat);
    if (ks.stride(1) != 1) ks = ks.contiguous();
    Tensor scores = empty({batch, m, n}, at::kFloat, q);
    check(p_rt_fp8_index_batched(q3.data_ptr(), data<float>(w3), k3.data_ptr(), data<float>(ks), data<float>(scores),
                                 batch, m, h, n, d, scores.stride(1), causal_offset.value_or(-1),
                                 batch > 1 ? k3.stride(0) / d : n, batch > 1 ? ks.stride(0) : n, scores.stride(0),
                                 stream()),
          "rt_fp8_index_batched");
    return lead ? scores : scores.reshape({m, n});
}

Tensor index_topk(const Tensor& scores, int64_t topk) {
    require_cuda({&scores});
    if (scores.scalar_type() != at::kFloat) fail("index_topk: scores must be float32");
    const int64_t n = scores.size(-1);
    Tensor s2 = scores.reshape({-1, n});
    if (s2.stride(1) != 1) s2 = s2.contiguous();
    const int64_t kk = std::min(topk, n);
    Tensor out = empty({s2.size(0), kk}, at::kInt, scores);
    check(p_rt_index_topk(data<float>(s2), data<int32_t>(out), s2.size(0), n, s2.stride(0), kk, stream()),
          "rt_index_topk");
    return out.reshape(with_last(scores, kk));
}

Tensor mla_sparse_decode(const Tensor& q_abs, const Tensor& q_pe, const Tensor& kv_cache, const Tensor& pe_cache,
                         const OptTensor& indices_in, double softmax_scale) {
    require_cuda({&q_abs});
    const std::pair<const char*, const Tensor*> named[] = {
        {"q_abs", &q_abs}, {"q_pe", &q_pe}, {"kv_cache", &kv_cache}, {"pe_cache", &pe_cache}};
    for (const auto& [name, t] : named)
        if (t->scalar_type() != at::kBFloat16 || t->dim() != 3 || t->stride(2) != 1)
            fail(std::string("mla_sparse_decode: ") + name + " must be bf16 [*, *, d] with a contiguous last dim");
    const int64_t batch = q_abs.size(0), heads = q_abs.size(1), keys = kv_cache.size(1);
    if (q_abs.size(2) != 512 || kv_cache.size(2) != 512 || !same_shape(q_pe, {batch, heads, 64}) ||
        !same_shape(pe_cache, {batch, keys, 64}) || kv_cache.size(0) != batch)
        fail("mla_sparse_decode: shapes must be [B,H,512], [B,H,64], [B,S,512], [B,S,64]");
    OptTensor indices = indices_in;
    int64_t n_sel = keys;
    if (indices) {
        if (indices->scalar_type() != at::kInt || indices->dim() != 2 || indices->size(0) != batch)
            fail("mla_sparse_decode: indices must be int32 [B, n_sel]");
        if (indices->stride(1) != 1) indices = indices->contiguous();
        n_sel = indices->size(1);
    }
    const int64_t splits = p_rt_mla_sparse_decode_splits(batch, heads, n_sel);
    Tensor out = empty({batch, heads, 512}, at::kBFloat16, q_abs);
    Tensor part_o = empty({batch * splits * heads * 512}, at::kFloat, q_abs);
    Tensor part_ml = empty({batch * splits * heads * 2}, at::kFloat, q_abs);
    check(p_rt_mla_sparse_decode(q_abs.data_ptr(), q_pe.data_ptr(), kv_cache.data_ptr(), pe_cache.data_ptr(),
                                 data<int32_t>(indices), out.data_ptr(), data<float>(part_o), data<float>(part_ml),
                                 batch, heads, keys, n_sel, q_abs.stride(0), q_abs.stride(1), q_pe.stride(0),
                                 q_pe.stride(1), kv_cache.stride(0), kv_cache.stride(1), pe_cache.stride(0),
                                 pe_cache.stride(1), indices ? indices->stride(0) : 0, splits,
                                 static_cast<float>(softmax_scale), stream()),
          "rt_mla_sparse_decode");
    return out;
}

}  // namespace

PYBIND11_MODULE(_rt_torch, m) {
    m.def("bind", &bind);
    m.def("table", [] {
        std::vector<std::string> names;
#define RT_NAME(name) names.emplace_back(#name);
        RT_TABLE(RT_NAME)
#undef RT_NAME
        return names;
    });
    // Other Python threads run while a call checks, allocates and launches: a launch may block on a full
    // queue (as behind a ctypes call, which lets go of the interpreter too).
#define RT_DEF(name) m.def(#name, &name, py::call_guard<py::gil_scoped_release>())
    RT_DEF(residual_norm);
    RT_DEF(rms_norm);
    RT_DEF(norm_rope);
    RT_DEF(rope);
    RT_DEF(swiglu);
    RT_DEF(act_quant);
    RT_DEF(swiglu_quant);
    RT_DEF(tensor_absmax);
    RT_DEF(swiglu_absmax);
    RT_DEF(nvfp4_quant);
    RT_DEF(linear_bf16);
    RT_DEF(linear_bf16_batched);
    RT_DEF(linear_fp8);
    RT_DEF(gemm_nvfp4_grouped);
    RT_DEF(moe_route);
    RT_DEF(moe_permute);
    RT_DEF(moe_tile_map);
    RT_DEF(moe_gather_nvfp4);
    RT_DEF(moe_quant_nvfp4);
    RT_DEF(moe_combine);
    RT_DEF(moe_experts);
    RT_DEF(index_prep);
    RT_DEF(index_head_weights);
    RT_DEF(fp8_index);
    RT_DEF(index_topk);
    RT_DEF(mla_sparse_decode);
#undef RT_DEF
}

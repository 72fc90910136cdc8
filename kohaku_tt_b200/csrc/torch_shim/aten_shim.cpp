// The aten fused-SDPA overloads on the CUDA key, registered from C++: the counterpart of the
// reference's TORCH_LIBRARY_IMPL block (aten_attention.cpp:959-974; tt_sdpa_overrideable
// :389-713, its backward :715-812, fused_refusal :62-127, tt_fused_sdp_choice :194-219).
//
// A thin shim: it checks the call with the reference's refusal rules, lets torch allocate
// the outputs in the layout each overload's meta kernel promises, fills a
// ktt_b200_attn_args block with raw pointers and element strides and calls the C ABI of
// libktt_b200.so on torch's current stream. Nothing here computes.
//
// Registration is dynamic (ktt_b200_aten_install / _uninstall create and destroy the
// torch::Library objects), so that a process can take the overloads out again.
//
// The file is also a Python extension module (`ktt_b200_native`): the eager fast paths of
// F.scaled_dot_product_attention, sdpa(key_lengths=), sdpa_varlen and decode_step. Small calls are
// bound by the host: through torch's composite (its backend choice, the conversion of a bool
// mask to a padded additive one by three kernels), Python custom operators, Python autograd
// functions and ctypes argument blocks they took 13, 57, 150 and 50 us a call.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/scaled_dot_product_attention_native.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>

#include "../../../include/ktt_b200.h"

namespace {

using at::Tensor;

// ---- the kernel scope of the calling thread (kohaku_tt_b200.sdpa_kernel) -------------------
thread_local int g_kernel = KTT_B200_KERNEL_AUTO;   // -1: the scope allows no kernel
thread_local std::string g_scope_names;             // empty outside a scope

// The first condition a call fails, or null (fused_refusal, aten_attention.cpp:62-127, minus
// the rules that only describe Tensix limits).
const char* fused_refusal(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask,
                          double dropout_p, bool is_causal) {
    const bool grads = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
    for (const Tensor* t : {&q, &k, &v}) {
        const bool ok_dtype = t->scalar_type() == at::kBFloat16 || (t->scalar_type() == at::kFloat && !grads);
        if (t->dim() != 4 || t->numel() == 0 || !ok_dtype || t->scalar_type() != q.scalar_type()) {
            return "q, k and v must be non-empty 4-D bf16 (fp32 without gradients)";
        }
    }
    if (dropout_p != 0.0) return "dropout";
    if (k.size(3) != q.size(3)) return "q and k need one head dim";
    if (k.size(0) != q.size(0) || v.size(0) != q.size(0) || v.size(1) != k.size(1) || q.size(1) % k.size(1) != 0 ||
        v.size(2) != k.size(2)) {
        return "q, k and v shapes do not match (K / V heads must divide Q heads)";
    }
    if (std::max(q.size(3), v.size(3)) > 256) return "head dims above 256 are not taken";
    if (is_causal && mask.has_value() && mask->defined()) return "causal takes no mask";
    if (mask.has_value() && mask->defined()) {
        if (mask->dim() > 4) return "the mask must broadcast to [B, H, Sq, Sk]";
        const int64_t full[4] = {q.size(0), q.size(1), q.size(2), k.size(2)};
        for (int64_t i = 0; i < mask->dim(); ++i) {
            const int64_t s = mask->size(mask->dim() - 1 - i);
            if (s != 1 && s != full[3 - i]) return "the mask must broadcast to [B, H, Sq, Sk]";
        }
    }
    return nullptr;
}

std::string describe(const Tensor& t) {
    std::string s = "[";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + "] " + std::string(c10::toString(t.scalar_type()));
}

void checked(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask, double dropout_p,
             bool is_causal) {
    const char* why = fused_refusal(q, k, v, mask, dropout_p, is_causal);
    if (!why) {
        TORCH_CHECK(g_kernel >= 0, "kohaku_tt_b200.sdpa_kernel(", g_scope_names,
                    "): no device kernel is allowed and there is no math fallback");
        return;
    }
    if (!g_scope_names.empty()) {
        std::string m = "none";
        if (mask.has_value() && mask->defined()) m = (mask->scalar_type() == at::kBool ? "bool " : "additive ") + describe(*mask);
        TORCH_CHECK(false, "kohaku_tt_b200.sdpa_kernel(", g_scope_names, "): no allowed kernel takes attention q ", describe(q),
                    ", k ", describe(k), ", v ", describe(v), ", mask ", m, is_causal ? ", causal" : "", ": ", why);
    }
    TORCH_CHECK_NOT_IMPLEMENTED(
        false, "kohaku_tt_b200: fused attention refused: ", why,
        ". On CUDA PyTorch picks the fused overload itself, so a refused call cannot fall back to the math composite from "
        "here: wrap it in torch.nn.attention.sdpa_kernel(SDPBackend.MATH), or call kohaku_tt_b200.uninstall()");
}

void raise_status(int rc, const char* what) {
    if (rc == KTT_B200_OK) return;
    const std::string msg = std::string("kohaku_tt_b200.") + what + ": " + ktt_b200_last_error();
    if (rc == KTT_B200_ERR_UNSUPPORTED) TORCH_CHECK_NOT_IMPLEMENTED(false, msg);
    if (rc == KTT_B200_ERR_BAD_ARGUMENT) TORCH_CHECK_VALUE(false, msg);
    TORCH_CHECK(false, msg);
}

Tensor rows_contiguous(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }

void set3(int64_t* dst, const Tensor& t) {
    dst[0] = t.stride(0);
    dst[1] = t.stride(1);
    dst[2] = t.stride(2);
}

// Mask operand: dtype code and the strides of its view as [b, h, sq, sk] (0 where it broadcasts). A
// converted copy is kept alive by the caller through `keep`.
void mask_operand(ktt_b200_attn_args& a, const c10::optional<Tensor>& mask, int64_t b, int64_t h, int64_t sq, int64_t sk, Tensor& keep) {
    a.mask = nullptr;
    a.mask_dtype = KTT_B200_MASK_NONE;
    if (!mask.has_value() || !mask->defined()) return;
    Tensor m = *mask;
    int code;
    switch (m.scalar_type()) {
        case at::kBool: case at::kByte: code = KTT_B200_MASK_BOOL; break;
        case at::kBFloat16: code = KTT_B200_MASK_BF16; break;
        case at::kFloat: code = KTT_B200_MASK_F32; break;
        case at::kHalf: code = KTT_B200_MASK_F16; break;
        default: m = m.to(at::kFloat); code = KTT_B200_MASK_F32; break;
    }
    const int64_t full[4] = {b, h, sq, sk}, lead = 4 - m.dim();
    for (int64_t i = 0; i < 4; ++i) {
        const int64_t size = i < lead ? 1 : m.size(i - lead);
        TORCH_CHECK_VALUE(size == 1 || size == full[i], "kohaku_tt_b200: the mask must broadcast to [B, H, Sq, Sk]");
        a.mask_strides[i] = size == 1 ? 0 : m.stride(i - lead);
    }
    a.mask = m.data_ptr();
    a.mask_dtype = code;
    keep = m;
}

// An output or workspace straight from the CUDA allocator: the dispatcher's share of at::empty is
// more than half of its cost, and an attention call makes several.
Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& like) {
    return at::detail::empty_cuda(sizes, dtype, like.device(), c10::nullopt);
}

// Buffers whose head must be zero before the first use and is left zero by every kernel: one per
// (device, stream), since calls that share one must not overlap on the GPU. At most kMost of them
// are kept; dropping one gives it back to the caching allocator, which orders its next use behind
// the work of its stream.
class ZeroedPool {
public:
    // A buffer of at least `bytes`, its first `zeroed` bytes zero.
    Tensor get(int64_t bytes, int64_t zeroed, const Tensor& like, cudaStream_t stream) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(stream, &capture);
        if (capture != cudaStreamCaptureStatusNone) return fresh(bytes, zeroed, like, stream);   // the graph zeroes its own at every replay
        const std::pair<int, cudaStream_t> key(like.get_device(), stream);
        std::lock_guard<std::mutex> lock(mutex_);
        auto it = buffers_.find(key);
        if (it == buffers_.end() || it->second.numel() < bytes) {
            if (it == buffers_.end() && buffers_.size() >= kMost) buffers_.clear();
            it = buffers_.insert_or_assign(key, fresh(bytes, zeroed, like, stream)).first;
        }
        return it->second;
    }
    void clear() {
        std::lock_guard<std::mutex> lock(mutex_);
        buffers_.clear();
    }

private:
    static constexpr size_t kMost = 32;
    static Tensor fresh(int64_t bytes, int64_t zeroed, const Tensor& like, cudaStream_t stream) {
        Tensor t = empty_cuda({bytes}, at::kByte, like);
        C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, zeroed, stream));
        return t;
    }
    std::mutex mutex_;
    std::map<std::pair<int, cudaStream_t>, Tensor> buffers_;
};
// (Never destroyed: at process exit the CUDA context may be gone before static objects are.)
ZeroedPool& forward_pool() {
    static ZeroedPool* pool = new ZeroedPool;
    return *pool;
}
ZeroedPool& decode_pool() {
    static ZeroedPool* pool = new ZeroedPool;
    return *pool;
}

// The tcgen05 forward's workspace. Without a mask that has a row per query it is the counter the
// CTAs draw their tiles from, which the kernel leaves zero. A plan of such a mask is up to 1 GB and
// belongs to the call; where the device has no room for it the call goes without, to a kernel that
// reads the mask itself.
constexpr int64_t kCounterBytes = 256;
Tensor forward_workspace(const ktt_b200_attn_args& a, const Tensor& like, cudaStream_t stream) {
    const int64_t need = ktt_b200_sdpa_forward_workspace(&a);
    if (need <= 0) return Tensor();
    if (need > kCounterBytes) {
        try {
            return empty_cuda({need}, at::kByte, like);
        } catch (const c10::OutOfMemoryError&) {
            return Tensor();
        }
    }
    return forward_pool().get(kCounterBytes, kCounterBytes, like, stream);
}

void fill_common(ktt_b200_attn_args& a, const Tensor& q, const Tensor& k, const Tensor& v, bool is_causal, c10::optional<double> scale) {
    std::memset(&a, 0, sizeof(a));
    a.batch = static_cast<int32_t>(q.size(0));
    a.heads = static_cast<int32_t>(q.size(1));
    a.kv_heads = static_cast<int32_t>(k.size(1));
    a.sq = static_cast<int32_t>(q.size(2));
    a.sk = static_cast<int32_t>(k.size(2));
    a.d = static_cast<int32_t>(q.size(3));
    a.dv = static_cast<int32_t>(v.size(3));
    a.causal = is_causal ? KTT_B200_CAUSAL_TOP_LEFT : KTT_B200_CAUSAL_NONE;
    a.scale = static_cast<float>(scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(q.size(3))));
    a.kernel = g_kernel < 0 ? KTT_B200_KERNEL_AUTO : g_kernel;
    a.q = q.data_ptr();
    a.k = k.data_ptr();
    a.v = v.data_ptr();
    set3(a.q_strides, q);
    set3(a.k_strides, k);
    set3(a.v_strides, v);
}

// What a call has beyond q, k and v.
struct Extras {
    c10::optional<Tensor> mask;     // dense: broadcastable to [B, H, Sq, Sk]; packed: [Tk]
    Tensor lengths;                 // int32 [B] on the device
    Tensor cu_q, cu_k;              // packed: int32 [n + 1] on the device
    int64_t max_q = 0, max_k = 0;
    int32_t causal = KTT_B200_CAUSAL_NONE;
    c10::optional<double> scale;
    bool packed() const { return cu_q.defined(); }
};

// Operand strides: (batch, head, row) of a dense [B, H, S, D], (0, head, row) of a packed [T, H, D].
void set_strides(int64_t* dst, const Tensor& t) {
    if (t.dim() == 4) {
        set3(dst, t);
    } else {
        dst[0] = 0;
        dst[1] = t.stride(1);
        dst[2] = t.stride(0);
    }
}

void fill_args(ktt_b200_attn_args& a, const Tensor& q, const Tensor& k, const Tensor& v, const Extras& x, Tensor& keep) {
    if (!x.packed()) {
        fill_common(a, q, k, v, false, x.scale);
        a.causal = x.causal;
        mask_operand(a, x.mask, q.size(0), q.size(1), q.size(2), k.size(2), keep);
        if (x.lengths.defined()) a.key_lengths = x.lengths.data_ptr<int32_t>();
        return;
    }
    std::memset(&a, 0, sizeof(a));
    a.batch = static_cast<int32_t>(x.cu_q.numel() - 1);
    a.heads = static_cast<int32_t>(q.size(1));
    a.kv_heads = static_cast<int32_t>(k.size(1));
    a.sq = static_cast<int32_t>(std::max<int64_t>(x.max_q, 1));
    a.sk = static_cast<int32_t>(std::max<int64_t>(x.max_k, 1));
    a.total_q = q.size(0);
    a.total_k = k.size(0);
    a.d = static_cast<int32_t>(q.size(2));
    a.dv = static_cast<int32_t>(v.size(2));
    a.causal = x.causal;
    a.scale = static_cast<float>(x.scale.has_value() ? *x.scale : 1.0 / std::sqrt(static_cast<double>(q.size(2))));
    a.kernel = g_kernel < 0 ? KTT_B200_KERNEL_AUTO : g_kernel;
    a.q = q.data_ptr();
    a.k = k.data_ptr();
    a.v = v.data_ptr();
    set_strides(a.q_strides, q);
    set_strides(a.k_strides, k);
    set_strides(a.v_strides, v);
    a.cu_seqlens_q = x.cu_q.data_ptr<int32_t>();
    a.cu_seqlens_k = x.cu_k.data_ptr<int32_t>();
}

// lse: [B, H, rows], or [H, Tq] for a packed call.
void set_lse(ktt_b200_attn_args& a, const Tensor& lse) {
    a.lse = lse.data_ptr<float>();
    a.lse_strides[0] = lse.dim() == 3 ? lse.stride(0) : 0;
    a.lse_strides[1] = lse.stride(lse.dim() - 2);
    a.lse_strides[2] = 1;
}

// Forward into `out` (already allocated in the layout the caller promises); returns the lse.
Tensor run_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Extras& x, Tensor& out, bool need_lse, int64_t lse_rows) {
    const Tensor q = rows_contiguous(q_), k = rows_contiguous(k_), v = rows_contiguous(v_);
    c10::cuda::CUDAGuard guard(q.device());
    ktt_b200_attn_args a;
    Tensor keep;
    fill_args(a, q, k, v, x, keep);
    a.out = out.data_ptr();
    set_strides(a.out_strides, out);
    Tensor lse;
    if (need_lse) {
        lse = x.packed() ? empty_cuda({q.size(1), q.size(0)}, at::kFloat, q) : empty_cuda({q.size(0), q.size(1), lse_rows}, at::kFloat, q);
        set_lse(a, lse);
    }
    cudaStream_t stream = at::cuda::getCurrentCUDAStream();
    Tensor ws = forward_workspace(a, q, stream);
    if (ws.defined()) {
        a.workspace = ws.data_ptr();
        a.workspace_bytes = ws.numel();
    }
    raise_status(ktt_b200_sdpa_forward(&a, stream), "sdpa_forward");
    return lse;
}

Tensor run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask, bool is_causal,
                   c10::optional<double> scale, Tensor& out, bool need_lse, int64_t lse_rows) {
    Extras x;
    x.mask = mask;
    x.causal = is_causal ? KTT_B200_CAUSAL_TOP_LEFT : KTT_B200_CAUSAL_NONE;
    x.scale = scale;
    return run_forward(q, k, v, x, out, need_lse, lse_rows);
}

std::tuple<Tensor, Tensor, Tensor> run_backward(const Tensor& dout_, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                                                const Tensor& out_, const Tensor& lse, const Extras& x) {
    const Tensor q = rows_contiguous(q_), k = rows_contiguous(k_), v = rows_contiguous(v_);
    const Tensor dout = rows_contiguous(dout_), out = rows_contiguous(out_);
    TORCH_CHECK_VALUE(lse.scalar_type() == at::kFloat && lse.stride(-1) == 1, "kohaku_tt_b200: lse must be fp32 with unit row stride");
    c10::cuda::CUDAGuard guard(q.device());
    ktt_b200_attn_args a;
    Tensor keep;
    fill_args(a, q, k, v, x, keep);
    Tensor dq = empty_cuda(q.sizes(), q.scalar_type(), q), dk = empty_cuda(k.sizes(), k.scalar_type(), k), dv = empty_cuda(v.sizes(), v.scalar_type(), v);
    a.out = out.data_ptr();
    set_lse(a, lse);
    a.dout = dout.data_ptr();
    a.dq = dq.data_ptr();
    a.dk = dk.data_ptr();
    a.dv_out = dv.data_ptr();
    set_strides(a.out_strides, out);
    set_strides(a.dout_strides, dout);
    set_strides(a.dq_strides, dq);
    set_strides(a.dk_strides, dk);
    set_strides(a.dv_strides, dv);
    const int64_t nbytes = ktt_b200_sdpa_backward_workspace(&a);
    if (nbytes <= 0) raise_status(KTT_B200_ERR_UNSUPPORTED, "sdpa_backward");
    Tensor work = empty_cuda({nbytes}, at::kByte, q);
    a.workspace = work.data_ptr();
    a.workspace_bytes = nbytes;
    raise_status(ktt_b200_sdpa_backward(&a, at::cuda::getCurrentCUDAStream()), "sdpa_backward");
    return {dq, dk, dv};
}

std::tuple<Tensor, Tensor, Tensor> run_backward(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out,
                                                const Tensor& lse, const c10::optional<Tensor>& mask, bool is_causal, c10::optional<double> scale) {
    TORCH_CHECK_VALUE(lse.dim() == 3, "kohaku_tt_b200: lse must be fp32 [B, H, rows] with unit row stride");
    Extras x;
    x.mask = mask;
    x.causal = is_causal ? KTT_B200_CAUSAL_TOP_LEFT : KTT_B200_CAUSAL_NONE;
    x.scale = scale;
    return run_backward(dout, q, k, v, out, lse, x);
}

// Output laid out the way torch's meta kernels of the flash, cuDNN and overrideable overloads
// promise (empty_like(query): the query's stride order).
Tensor out_like(const Tensor& q, int64_t dv) {
    if (dv == q.size(3)) return at::empty_like(q);
    int order[4] = {0, 1, 2, 3};
    std::sort(order, order + 4, [&](int x, int y) { return q.stride(x) != q.stride(y) ? q.stride(x) > q.stride(y) : x < y; });
    const int64_t shape[4] = {q.size(0), q.size(1), q.size(2), dv};
    Tensor out = at::empty({shape[order[0]], shape[order[1]], shape[order[2]], shape[order[3]]}, q.options());
    int64_t perm[4];
    for (int i = 0; i < 4; ++i) perm[order[i]] = i;
    return out.permute({perm[0], perm[1], perm[2], perm[3]});
}

struct Bf16 {
    Tensor q, k, v;
    bool cast;
};

// fp32 inputs without gradients are cast at entry and the output cast back
// (aten_attention.cpp:400-415).
Bf16 as_bf16(const Tensor& q, const Tensor& k, const Tensor& v) {
    if (q.scalar_type() == at::kFloat) return {q.to(at::kBFloat16), k.to(at::kBFloat16), v.to(at::kBFloat16), true};
    return {q, k, v, false};
}

Tensor empty0(const Tensor& like, at::ScalarType dtype) { return at::empty({0}, like.options().dtype(dtype)); }

c10::optional<Tensor> bias_or_none(const Tensor& bias) {
    if (!bias.defined() || bias.numel() == 0) return c10::nullopt;
    return bias;
}

// Gradient of an additive bias: dS summed over the dims the bias broadcasts, recomputed with
// separate matmul / softmax steps as the reference's masked backward does
// (aten_attention.cpp:781-811).
Tensor bias_gradient(const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias,
                     c10::optional<double> scale) {
    const int64_t rep = q.size(1) / k.size(1);
    const Tensor kf = k.to(at::kFloat).repeat_interleave(rep, 1), vf = v.to(at::kFloat).repeat_interleave(rep, 1);
    const double sc = scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(q.size(3)));
    const Tensor s = at::matmul(q.to(at::kFloat), kf.transpose(-1, -2)) * sc + bias.to(at::kFloat).clamp_min(-5e5);
    const Tensor p = at::softmax(s, -1);
    const Tensor dp = at::matmul(grad_out.to(at::kFloat), vf.transpose(-1, -2));
    Tensor ds = p * (dp - (dp * p).sum(-1, true));
    Tensor b4 = bias;
    while (b4.dim() < 4) b4 = b4.unsqueeze(0);
    std::vector<int64_t> dims;
    for (int64_t i = 0; i < 4; ++i) {
        if (b4.size(i) == 1 && ds.size(i) != 1) dims.push_back(i);
    }
    if (!dims.empty()) ds = ds.sum(dims, true);
    return ds.reshape(bias.sizes()).to(bias.scalar_type());
}

// ---- the overloads ---------------------------------------------------------------------------

std::tuple<Tensor, Tensor, Tensor, Tensor, c10::SymInt, c10::SymInt, Tensor, Tensor, Tensor> flash_forward(
    const Tensor& q, const Tensor& k, const Tensor& v, double dropout_p, bool is_causal, bool /*return_debug_mask*/,
    c10::optional<double> scale) {
    checked(q, k, v, c10::nullopt, dropout_p, is_causal);
    const Bf16 x = as_bf16(q, k, v);
    Tensor out = out_like(x.q, x.v.size(3));
    Tensor lse = run_forward(x.q, x.k, x.v, c10::nullopt, is_causal, scale, out, true, q.size(2));
    if (x.cast) out = out.to(at::kFloat);
    // Dropout is refused, so nobody reads the generator state: left unwritten.
    return {out, lse, empty0(q, at::kLong), empty0(q, at::kLong), c10::SymInt(q.size(2)), c10::SymInt(k.size(2)),
            at::empty({2}, q.options().dtype(at::kUInt64)), at::empty({}, q.options().dtype(at::kUInt64)),
            empty0(q, q.scalar_type())};
}

std::tuple<Tensor, Tensor, Tensor> flash_backward(
    const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
    const Tensor&, const Tensor&, c10::SymInt, c10::SymInt, double dropout_p, bool is_causal, const Tensor&, const Tensor&,
    c10::optional<double> scale) {
    checked(q, k, v, c10::nullopt, dropout_p, is_causal);
    return run_backward(grad_out, q, k, v, out, lse, c10::nullopt, is_causal, scale);
}

std::tuple<Tensor, Tensor, Tensor, Tensor> efficient_forward(
    const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& bias, bool compute_lse, double dropout_p,
    bool is_causal, c10::optional<double> scale) {
    checked(q, k, v, bias, dropout_p, is_causal);
    const Bf16 x = as_bf16(q, k, v);
    // The efficient overload's meta promises [B, Sq, H, Dv] storage seen as [B, H, Sq, Dv].
    Tensor out = at::empty({q.size(0), q.size(2), q.size(1), v.size(3)}, x.q.options()).transpose(1, 2);
    const int64_t rows = (q.size(2) + 31) / 32 * 32;
    Tensor lse = run_forward(x.q, x.k, x.v, bias, is_causal, scale, out, compute_lse, rows);
    if (!lse.defined()) lse = at::empty({q.size(0), q.size(1), 0}, q.options().dtype(at::kFloat));
    if (x.cast) out = out.to(at::kFloat);
    return {out, lse, at::empty({}, q.options().dtype(at::kLong)), at::empty({}, q.options().dtype(at::kLong))};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> efficient_backward(
    const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias_, const Tensor& out,
    const Tensor& lse, const Tensor&, const Tensor&, double dropout_p, std::array<bool, 4> grad_input_mask, bool is_causal,
    c10::optional<double> scale) {
    const c10::optional<Tensor> bias = bias_or_none(bias_);
    checked(q, k, v, bias, dropout_p, is_causal);
    auto [dq, dk, dv] = run_backward(grad_out, q, k, v, out, lse, bias, is_causal, scale);
    Tensor dbias;
    if (bias.has_value() && grad_input_mask[3]) dbias = bias_gradient(grad_out, q, k, v, *bias, scale);
    return {dq, dk, dv, dbias};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, c10::SymInt, c10::SymInt, Tensor, Tensor, Tensor> cudnn_forward(
    const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& bias, bool /*compute_lse*/, double dropout_p,
    bool is_causal, bool /*return_debug_mask*/, c10::optional<double> scale) {
    checked(q, k, v, bias, dropout_p, is_causal);
    const Bf16 x = as_bf16(q, k, v);
    Tensor out = out_like(x.q, x.v.size(3));
    Tensor lse = run_forward(x.q, x.k, x.v, bias, is_causal, scale, out, true, q.size(2));
    if (x.cast) out = out.to(at::kFloat);
    return {out, lse.unsqueeze(-1), empty0(q, at::kLong), empty0(q, at::kLong), c10::SymInt(q.size(2)), c10::SymInt(k.size(2)),
            at::empty({}, q.options().dtype(at::kLong)), at::empty({}, q.options().dtype(at::kLong)), empty0(q, q.scalar_type())};
}

std::tuple<Tensor, Tensor, Tensor> cudnn_backward(
    const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse_,
    const Tensor&, const Tensor&, const Tensor& bias_, const Tensor&, const Tensor&, c10::SymInt, c10::SymInt, double dropout_p,
    bool is_causal, c10::optional<double> scale) {
    const c10::optional<Tensor> bias = bias_or_none(bias_);
    checked(q, k, v, bias, dropout_p, is_causal);
    const Tensor lse = (lse_.dim() == 4 ? lse_.squeeze(-1) : lse_).contiguous();
    return run_backward(grad_out, q, k, v, out, lse, bias, is_causal, scale);
}

std::tuple<Tensor, Tensor, Tensor, Tensor, c10::SymInt, c10::SymInt, Tensor, Tensor, Tensor> overrideable_forward(
    const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& bias, double dropout_p, bool is_causal,
    bool /*return_debug_mask*/, c10::optional<double> scale) {
    checked(q, k, v, bias, dropout_p, is_causal);
    const Bf16 x = as_bf16(q, k, v);
    Tensor out = out_like(x.q, x.v.size(3));
    Tensor lse = run_forward(x.q, x.k, x.v, bias, is_causal, scale, out, true, q.size(2));
    if (x.cast) out = out.to(at::kFloat);
    return {out, lse, empty0(q, at::kLong), empty0(q, at::kLong), c10::SymInt(q.size(2)), c10::SymInt(k.size(2)),
            at::empty({}, q.options().dtype(at::kLong)), at::empty({}, q.options().dtype(at::kLong)), empty0(q, q.scalar_type())};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> overrideable_backward(
    const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias_,
    std::array<bool, 4> grad_input_mask, const Tensor& out, const Tensor& lse, const Tensor&, const Tensor&, c10::SymInt,
    c10::SymInt, double dropout_p, bool is_causal, const Tensor&, const Tensor&, c10::optional<double> scale) {
    const c10::optional<Tensor> bias = bias_or_none(bias_);
    checked(q, k, v, bias, dropout_p, is_causal);
    auto [dq, dk, dv] = run_backward(grad_out, q, k, v, out, lse, bias, is_causal, scale);
    Tensor dbias = empty0(q, q.scalar_type());
    if (bias.has_value() && grad_input_mask[3]) dbias = bias_gradient(grad_out, q, k, v, *bias, scale);
    return {dq, dk, dv, dbias};
}

// SDPBackend: MATH 0, OVERRIDEABLE 4. MATH when torch's own switch has every fused backend
// whose overload lands here turned off (the reference asks the one switch its overload sits
// behind, aten_attention.cpp:204-207), or when the shapes are refused.
int64_t fused_sdp_choice(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask, double dropout_p,
                         bool is_causal, c10::optional<double> /*scale*/, bool /*enable_gqa*/) {
    auto& ctx = at::globalContext();
    if (!(ctx.userEnabledFlashSDP() || ctx.userEnabledMemEfficientSDP() || ctx.userEnabledCuDNNSDP() || ctx.userEnabledOverrideableSDP())) {
        return 0;
    }
    return fused_refusal(q, k, v, mask, dropout_p, is_causal) ? 0 : 4;
}

// ---- eager fast paths ------------------------------------------------------------------------
//
// They take plain CUDA tensors outside of every mode that wants to see the call itself (tracing,
// fake tensors, functorch, dispatch and function modes); anything else goes the way it always
// went, through torch's composite or the registered operators.

constexpr c10::DispatchKeySet kPlainKeys({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA});

bool plain(const Tensor& t) {
    return t.is_cuda() && !(t.key_set().raw_repr() & ~kPlainKeys.raw_repr()) && !t._fw_grad(0).defined();   // (set difference would keep the backend bits)
}

bool eager() {
    const c10::DispatchKeySet modes({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                     c10::DispatchKey::PreDispatch, c10::DispatchKey::Python, c10::DispatchKey::Functionalize});
    return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes);
}

bool wants_grad(const Tensor& q, const Tensor& k, const Tensor& v) {
    return at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
}

// Output [B, H, Sq, Dv] laid out [B, Sq, H, Dv] when q is a head view of a [B, S, H * D] storage
// (the reference's pitched route, aten_attention.cpp:605-628), else contiguous.
Tensor out_like_query(const Tensor& q, int64_t dv) {
    const int64_t b = q.size(0), h = q.size(1), s = q.size(2), d = q.size(3);
    if (h > 1 && s > 1 && q.stride(1) == d && q.stride(2) >= h * d) return empty_cuda({b, s, h, dv}, q.scalar_type(), q).transpose(1, 2);
    return empty_cuda({b, h, s, dv}, q.scalar_type(), q);
}

// A gradient the kernels can read: unit row stride, no broadcast dims.
Tensor readable(const Tensor& g) {
    for (int64_t i = 0; i < g.dim(); ++i) {
        if (g.size(i) > 1 && g.stride(i) == 0) return g.contiguous();
    }
    return rows_contiguous(g);
}

// An allocated output on its way through Function::apply (a bare tensor would be an input of the node).
struct Allocated {
    Tensor t;
};

// Autograd node of the fast paths. q, k, v, the output, its row statistics and the device-side
// extras are saved; only q, k and v get a gradient.
struct Attention : torch::autograd::Function<Attention> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Extras& x, const Allocated& to) {
        at::AutoDispatchBelowADInplaceOrView guard;
        Tensor out = to.t;
        Tensor lse = run_forward(q, k, v, x, out, true, x.packed() ? 0 : q.size(2));
        const Tensor none;
        ctx->save_for_backward({q, k, v, out, lse, x.mask.has_value() ? *x.mask : none, x.lengths, x.cu_q, x.cu_k});
        ctx->saved_data["sizes"] = std::vector<int64_t>{x.causal, x.max_q, x.max_k};
        if (x.scale.has_value()) ctx->saved_data["scale"] = *x.scale;
        return out;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const auto sizes = ctx->saved_data["sizes"].toIntVector();
        Extras x;
        if (saved[5].defined()) x.mask = saved[5];
        x.lengths = saved[6];
        x.cu_q = saved[7];
        x.cu_k = saved[8];
        x.causal = static_cast<int32_t>(sizes[0]);
        x.max_q = sizes[1];
        x.max_k = sizes[2];
        const auto scale = ctx->saved_data.find("scale");
        if (scale != ctx->saved_data.end()) x.scale = scale->second.toDouble();
        if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        torch::autograd::variable_list out;
        {
            at::AutoDispatchBelowADInplaceOrView guard;
            auto [dq, dk, dv] = run_backward(readable(grads[0]), saved[0], saved[1], saved[2], saved[3], saved[4], x);
            out = {dq, dk, dv};
        }
        if (at::GradMode::is_enabled()) {   // create_graph: differentiating the gradients is an error, not a silent zero
            for (Tensor& g : out) g.set_requires_grad(true);   // (a node is only attached to what may need one)
            out = (*std::make_shared<torch::autograd::DelayedError>("kohaku_tt_b200: the gradients of attention are not differentiable", 3))(std::move(out));
        }
        return {out[0], out[1], out[2], Tensor(), Tensor()};
    }
};

// aten::scaled_dot_product_attention itself. torch's composite asks its own chooser, which for bf16
// CUDA tensors of these head dims lands in this file's cuDNN or flash overload in any case (both
// return a tensor laid out like the query); calls it would send elsewhere, refuse or convert first
// (fp32, dropout, other head dims, a mask that wants a gradient, a backend switched off) go to it.
bool direct_sdpa(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask, double dropout_p, bool is_causal, bool enable_gqa) {
    if (g_kernel < 0 || !eager() || !plain(q) || !plain(k) || !plain(v)) return false;
    if (q.scalar_type() != at::kBFloat16 || q.dim() != 4 || q.size(3) % 8 || q.size(3) > 128 || v.dim() != 4 || v.size(3) != q.size(3)) return false;
    if (q.device() != k.device() || q.device() != v.device()) return false;
    if (fused_refusal(q, k, v, mask, dropout_p, is_causal) || (!enable_gqa && q.size(1) != k.size(1))) return false;
    if (mask.has_value() && mask->defined()) {
        const Tensor& m = *mask;
        if (!plain(m) || m.requires_grad() || m.device() != q.device()) return false;
        if (m.scalar_type() != at::kBool && m.scalar_type() != at::kBFloat16 && m.scalar_type() != at::kFloat) return false;
    }
    const auto& ctx = at::globalContext();
    return ctx.userEnabledFlashSDP() && ctx.userEnabledMemEfficientSDP() && ctx.userEnabledCuDNNSDP();
}

Tensor sdpa_entry(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& mask, double dropout_p, bool is_causal,
                  c10::optional<double> scale, bool enable_gqa) {
    if (!direct_sdpa(q, k, v, mask, dropout_p, is_causal, enable_gqa)) {
        return at::native::scaled_dot_product_attention(q, k, v, mask, dropout_p, is_causal, scale, enable_gqa);
    }
    Extras x;
    if (mask.has_value() && mask->defined()) x.mask = mask;
    x.causal = is_causal ? KTT_B200_CAUSAL_TOP_LEFT : KTT_B200_CAUSAL_NONE;
    x.scale = scale;
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView guard;
        out = q.is_contiguous() ? empty_cuda(q.sizes(), at::kBFloat16, q) : at::empty_like(q);
    }
    if (wants_grad(q, k, v)) return Attention::apply(q, k, v, x, Allocated{out});
    run_forward(q, k, v, x, out, false, 0);
    return out;
}

// Decode: what the split-K kernel takes (ops.decode_takes).
bool decode_takes(const Tensor& q, const Tensor& k, const Tensor& v) {
    const int64_t h = q.size(1), hk = k.size(1), d = q.size(3);
    if (hk == 0 || h % hk || v.size(3) != d || (d != 64 && d != 128) || (h / hk) * q.size(2) > 16 || q.size(0) > 512) return false;
    if (q.stride(3) != 1 || k.stride(3) != 1 || v.stride(3) != 1) return false;
    for (int i = 0; i < 3; ++i) {
        if (k.stride(i) % 8 || v.stride(i) % 8 || q.stride(i) % 2) return false;
    }
    return !((reinterpret_cast<uintptr_t>(k.data_ptr()) | reinterpret_cast<uintptr_t>(v.data_ptr())) & 15) && !(reinterpret_cast<uintptr_t>(q.data_ptr()) & 3);
}

// Fields and scratch of a decode call; the scratch starts with 1,024 int32 ticket counters.
Tensor fill_decode(ktt_b200_decode_args& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lengths, const Tensor& out,
                   c10::optional<double> scale, cudaStream_t stream) {
    a.batch = static_cast<int32_t>(q.size(0));
    a.heads = static_cast<int32_t>(q.size(1));
    a.kv_heads = static_cast<int32_t>(k.size(1));
    a.sq = static_cast<int32_t>(q.size(2));
    a.sk = static_cast<int32_t>(k.size(2));
    a.d = a.dv = static_cast<int32_t>(q.size(3));
    a.scale = static_cast<float>(scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(q.size(3))));
    a.q = q.data_ptr();
    a.k = k.data_ptr();
    a.v = v.data_ptr();
    a.out = out.data_ptr();
    set3(a.q_strides, q);
    set3(a.k_strides, k);
    set3(a.v_strides, v);
    set3(a.out_strides, out);
    a.key_lengths = lengths.data_ptr<int32_t>();
    const int64_t need = ktt_b200_decode_scratch_bytes(&a);
    if (need <= 0) raise_status(KTT_B200_ERR_UNSUPPORTED, "decode");
    Tensor scratch = decode_pool().get(need, 4096, q, stream);
    a.scratch = scratch.data_ptr();
    a.scratch_bytes = need;
    return scratch;
}

// Same dtype, device and shapes that go together (the checks of ops._dense_args).
bool dense_ok(const Tensor& q, const Tensor& k, const Tensor& v) {
    if (!plain(q) || !plain(k) || !plain(v) || q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return false;
    if (q.scalar_type() != at::kBFloat16 || k.scalar_type() != at::kBFloat16 || v.scalar_type() != at::kBFloat16) return false;
    if (q.device() != k.device() || q.device() != v.device() || q.numel() == 0 || k.numel() == 0 || v.numel() == 0) return false;
    return k.size(0) == q.size(0) && v.size(0) == q.size(0) && k.size(1) == v.size(1) && k.size(2) == v.size(2) && k.size(3) == q.size(3);
}

bool int32_vector(const Tensor& t, const Tensor& like, int64_t n) {
    return plain(t) && t.scalar_type() == at::kInt && t.dim() == 1 && t.numel() == n && t.is_contiguous() && t.device() == like.device();
}

// ---- Python ------------------------------------------------------------------------------------

const Tensor* tensor_of(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

bool scale_of(PyObject* o, c10::optional<double>& scale) {
    if (o == Py_None) return true;
    const double x = PyFloat_AsDouble(o);
    if (x == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    scale = x;
    return true;
}

// A fast path that the library refuses gives the call back: the general path words the refusal.
template <typename F>
bool attempted(F&& call) {
    try {
        call();
        return true;
    } catch (const c10::NotImplementedError&) {
        return false;
    }
}

bool callable_now() { return g_kernel >= 0 && !at::impl::torch_function_mode_enabled() && eager(); }

// sdpa_lengths(q, k, v, lengths, is_causal, scale): kohaku_tt_b200.sdpa with device lengths, or None
// when the call is not one for the fast path.
PyObject* py_sdpa_lengths(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const Tensor *q, *k, *v, *len;
    Extras x;
    if (n != 6 || !callable_now() || !(q = tensor_of(args[0])) || !(k = tensor_of(args[1])) || !(v = tensor_of(args[2])) ||
        !(len = tensor_of(args[3])) || !scale_of(args[5], x.scale) || !dense_ok(*q, *k, *v) || !int32_vector(*len, *q, q->size(0))) Py_RETURN_NONE;
    const bool causal = args[4] == Py_True;
    x.lengths = *len;
    x.causal = causal ? KTT_B200_CAUSAL_TOP_LEFT : KTT_B200_CAUSAL_NONE;
    Tensor out;
    const bool done = attempted([&] {
        pybind11::gil_scoped_release release;
        if (wants_grad(*q, *k, *v)) {
            out = Attention::apply(*q, *k, *v, x, Allocated{out_like_query(*q, v->size(3))});
        } else {
            at::AutoDispatchBelowADInplaceOrView guard;
            if (!causal && decode_takes(*q, *k, *v)) {
                c10::cuda::CUDAGuard device(q->device());
                cudaStream_t stream = at::cuda::getCurrentCUDAStream();
                out = empty_cuda(q->sizes(), at::kBFloat16, *q);
                ktt_b200_decode_args a;
                std::memset(&a, 0, sizeof(a));
                const Tensor scratch = fill_decode(a, *q, *k, *v, *len, out, x.scale, stream);
                raise_status(ktt_b200_decode(&a, stream), "decode");
            } else {
                out = out_like_query(*q, v->size(3));
                run_forward(*q, *k, *v, x, out, false, 0);
            }
        }
    });
    if (!done) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// decode_step(q, k_new, v_new, k_cache, v_cache, lengths, cos, sin, scale, lengths_out): the output,
// or None when the call is not one for the fast path (ops.decode_append then says what it wants).
PyObject* py_decode_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10 || !callable_now()) Py_RETURN_NONE;
    const Tensor* t[8];
    for (int i = 0; i < 8; ++i) {
        if (!(t[i] = tensor_of(args[i])) || !plain(*t[i])) Py_RETURN_NONE;
    }
    const Tensor &q = *t[0], &kn = *t[1], &vn = *t[2], &k = *t[3], &v = *t[4], &len = *t[5], &cos = *t[6], &sin = *t[7];
    c10::optional<double> scale;
    if (!scale_of(args[8], scale) || !dense_ok(q, k, v) || q.size(2) != 1 || !decode_takes(q, k, v) || !int32_vector(len, q, q.size(0))) Py_RETURN_NONE;
    const int64_t b = q.size(0), hk = k.size(1), d = q.size(3);
    for (const Tensor* r : {&kn, &vn}) {
        if (r->scalar_type() != at::kBFloat16 || r->device() != q.device() || r->dim() != 4 || r->size(0) != b || r->size(1) != hk || r->size(2) != 1 ||
            r->size(3) != d || r->stride(3) != 1) Py_RETURN_NONE;
    }
    for (const Tensor* r : {&cos, &sin}) {
        if (r->scalar_type() != at::kBFloat16 || r->device() != q.device() || r->dim() != 2 || r->size(1) != d || r->stride(1) != 1 ||
            r->size(0) != cos.size(0) || r->stride(0) != cos.stride(0)) Py_RETURN_NONE;
    }
    const bool by_position = cos.size(0) != b;
    if (by_position && cos.size(0) < k.size(2)) Py_RETURN_NONE;
    const Tensor* len_out = nullptr;
    if (args[9] != Py_None && (!(len_out = tensor_of(args[9])) || !int32_vector(*len_out, q, b))) Py_RETURN_NONE;
    Tensor out;
    const bool done = attempted([&] {
        pybind11::gil_scoped_release release;
        at::AutoDispatchBelowADInplaceOrView guard;
        c10::cuda::CUDAGuard device(q.device());
        cudaStream_t stream = at::cuda::getCurrentCUDAStream();
        out = empty_cuda(q.sizes(), at::kBFloat16, q);
        ktt_b200_decode_append_args app;
        std::memset(&app, 0, sizeof(app));
        const Tensor scratch = fill_decode(app.base, q, k, v, len, out, scale, stream);
        app.k_new = kn.data_ptr();
        app.v_new = vn.data_ptr();
        for (int i = 0; i < 2; ++i) {
            app.k_new_strides[i] = kn.stride(i);
            app.v_new_strides[i] = vn.stride(i);
        }
        app.cos = cos.data_ptr();
        app.sin = sin.data_ptr();
        app.rope_row_stride = cos.stride(0);
        app.rope_by_position = by_position ? 1 : 0;
        if (len_out) app.lengths_out = len_out->data_ptr<int32_t>();
        raise_status(ktt_b200_decode_append(&app, stream), "decode_append");
    });
    if (!done) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// Offsets on the host: a contiguous int32 or int64 CPU tensor.
bool host_offsets(PyObject* o, std::vector<int32_t>& out) {
    const Tensor* t = tensor_of(o);
    if (!t || !t->device().is_cpu() || t->dim() != 1 || !t->is_contiguous() || t->numel() < 2 || t->requires_grad()) return false;
    const int64_t n = t->numel();
    out.resize(n);
    if (t->scalar_type() == at::kInt) {
        std::memcpy(out.data(), t->data_ptr<int32_t>(), n * sizeof(int32_t));
    } else if (t->scalar_type() == at::kLong) {
        const int64_t* p = t->data_ptr<int64_t>();
        for (int64_t i = 0; i < n; ++i) {
            if (p[i] < 0 || p[i] > INT32_MAX) return false;
            out[i] = static_cast<int32_t>(p[i]);
        }
    } else {
        return false;
    }
    return true;
}

// Both offset vectors in one copy to the device (queries first). The host side is staged by the
// driver (a copy of less than 64 KB from pageable memory), so the vectors may go at once.
Tensor offsets_to_device(const std::vector<int32_t>& cu_q, const std::vector<int32_t>& cu_k, bool same, const Tensor& like) {
    std::vector<int32_t> both(cu_q);
    if (!same) both.insert(both.end(), cu_k.begin(), cu_k.end());
    Tensor dev = empty_cuda({static_cast<int64_t>(both.size())}, at::kInt, like);
    C10_CUDA_CHECK(cudaMemcpyAsync(dev.data_ptr(), both.data(), both.size() * sizeof(int32_t), cudaMemcpyHostToDevice, at::cuda::getCurrentCUDAStream()));
    return dev;
}

// sdpa_varlen(q, k, v, cu_q, cu_k or None, max_q or None, max_k or None, is_causal, scale), offsets
// on the host and no mask: the output, or None when the call is not one for the fast path
// (offsets that break a rule among them: attention.check_offsets then says which; a stream that
// captures: torch then refuses the copy of the offsets).
PyObject* py_sdpa_varlen(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const Tensor *q, *k, *v;
    Extras x;
    std::vector<int32_t> cq, ck;
    if (n != 9 || !callable_now() || !(q = tensor_of(args[0])) || !(k = tensor_of(args[1])) || !(v = tensor_of(args[2])) ||
        !scale_of(args[8], x.scale) || !host_offsets(args[3], cq) || (args[4] != Py_None && !host_offsets(args[4], ck))) Py_RETURN_NONE;
    const bool given_k = args[4] != Py_None;
    if (!given_k) ck = cq;
    for (const Tensor* t : {q, k, v}) {
        if (!plain(*t) || t->dim() != 3 || t->numel() == 0 || t->scalar_type() != at::kBFloat16 || t->device() != q->device()) Py_RETURN_NONE;
    }
    if (k->size(0) != v->size(0) || k->size(1) != v->size(1) || k->size(2) != q->size(2)) Py_RETURN_NONE;
    {
        // A captured copy would read the offsets again at every replay, long after this call's are gone.
        c10::cuda::CUDAGuard device(q->device());
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        C10_CUDA_CHECK(cudaStreamIsCapturing(at::cuda::getCurrentCUDAStream(), &capture));
        if (capture != cudaStreamCaptureStatusNone) Py_RETURN_NONE;
    }
    const bool causal = args[7] == Py_True, same = !given_k || cq == ck;
    if (cq.size() != ck.size() || cq[0] != 0 || ck[0] != 0 || cq.back() != q->size(0) || ck.back() != k->size(0)) Py_RETURN_NONE;
    int32_t longest_q = 0, longest_k = 0;
    for (size_t i = 0; i + 1 < cq.size(); ++i) {
        const int32_t lq = cq[i + 1] - cq[i], lk = ck[i + 1] - ck[i];
        if (lq < 0 || lk < 0 || (lq > 0 && lk == 0) || (causal && lq > lk)) Py_RETURN_NONE;
        longest_q = std::max(longest_q, lq);
        longest_k = std::max(longest_k, lk);
    }
    x.max_q = longest_q;
    x.max_k = longest_k;
    for (int i = 0; i < 2; ++i) {
        if (args[5 + i] == Py_None) continue;
        const long given = PyLong_AsLong(args[5 + i]);
        if (given == -1 && PyErr_Occurred()) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        (i ? x.max_k : x.max_q) = given;
    }
    x.causal = causal ? KTT_B200_CAUSAL_BOTTOM_RIGHT : KTT_B200_CAUSAL_NONE;
    Tensor out;
    const bool done = attempted([&] {
        pybind11::gil_scoped_release release;
        c10::cuda::CUDAGuard device(q->device());
        const Tensor dev = offsets_to_device(cq, ck, same, *q);
        const int64_t count = static_cast<int64_t>(cq.size());
        {
            at::AutoDispatchBelowADInplaceOrView guard;
            x.cu_q = dev.narrow(0, 0, count);
            x.cu_k = same ? x.cu_q : dev.narrow(0, count, count);
            out = empty_cuda({q->size(0), q->size(1), v->size(2)}, at::kBFloat16, *q);
        }
        if (wants_grad(*q, *k, *v)) {
            out = Attention::apply(*q, *k, *v, x, Allocated{out});
        } else {
            at::AutoDispatchBelowADInplaceOrView guard;
            run_forward(*q, *k, *v, x, out, false, 0);
        }
    });
    if (!done) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

PyObject* py_drop_workspaces(PyObject*, PyObject*) {
    forward_pool().clear();
    decode_pool().clear();
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"sdpa_lengths", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sdpa_lengths)), METH_FASTCALL, nullptr},
    {"decode_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_decode_step)), METH_FASTCALL, nullptr},
    {"sdpa_varlen", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sdpa_varlen)), METH_FASTCALL, nullptr},
    {"drop_workspaces", py_drop_workspaces, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "ktt_b200_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

std::unique_ptr<torch::Library> g_autograd_library;
std::unique_ptr<torch::Library> g_library;
std::mutex g_install_mutex;

}  // namespace

extern "C" {

__attribute__((visibility("default"))) int ktt_b200_aten_install(void) {
    std::lock_guard<std::mutex> lock(g_install_mutex);
    if (g_library) return 0;
    try {
        auto lib = std::make_unique<torch::Library>(torch::Library::IMPL, "aten", c10::make_optional(c10::DispatchKey::CUDA), __FILE__, __LINE__);
        lib->impl("_scaled_dot_product_flash_attention", TORCH_FN(flash_forward));
        lib->impl("_scaled_dot_product_flash_attention_backward", TORCH_FN(flash_backward));
        lib->impl("_scaled_dot_product_efficient_attention", TORCH_FN(efficient_forward));
        lib->impl("_scaled_dot_product_efficient_attention_backward", TORCH_FN(efficient_backward));
        lib->impl("_scaled_dot_product_cudnn_attention", TORCH_FN(cudnn_forward));
        lib->impl("_scaled_dot_product_cudnn_attention_backward", TORCH_FN(cudnn_backward));
        lib->impl("_scaled_dot_product_fused_attention_overrideable", TORCH_FN(overrideable_forward));
        lib->impl("_scaled_dot_product_fused_attention_overrideable_backward", TORCH_FN(overrideable_backward));
        lib->impl("_fused_sdp_choice", TORCH_FN(fused_sdp_choice));
        lib->impl("scaled_dot_product_attention", TORCH_FN(sdpa_entry));
        auto grad = std::make_unique<torch::Library>(torch::Library::IMPL, "aten", c10::make_optional(c10::DispatchKey::AutogradCUDA), __FILE__, __LINE__);
        grad->impl("scaled_dot_product_attention", TORCH_FN(sdpa_entry));
        g_library = std::move(lib);
        g_autograd_library = std::move(grad);
    } catch (const std::exception&) {
        return -1;
    }
    return 0;
}

__attribute__((visibility("default"))) int ktt_b200_aten_uninstall(void) {
    std::lock_guard<std::mutex> lock(g_install_mutex);
    g_autograd_library.reset();
    g_library.reset();
    return 0;
}

__attribute__((visibility("default"))) PyObject* PyInit_ktt_b200_native(void) { return PyModule_Create(&g_module); }

// The calling thread's kernel scope: `kernel` is a KTT_B200_KERNEL_* code or -1 (the scope
// allows no kernel); `names` the scope's kernel list for error messages ("" outside a scope).
__attribute__((visibility("default"))) void ktt_b200_aten_set_scope(int kernel, const char* names) {
    g_kernel = kernel;
    g_scope_names = names ? names : "";
}

}  // extern "C"

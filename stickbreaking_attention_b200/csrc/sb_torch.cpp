// Native host path of the PyTorch layer: argument checks, allocation of results and workspaces, the C-ABI calls and the autograd
// node, so that a call costs one Python -> C++ transition instead of ~60 Python-level operations.  For small problems the host
// is what bounds a step: forward + backward of 2048 tokens took 201 us through the Python layer, of which the kernels
// were 66 us.  Behaviour is that of ops.py, which keeps the traced (torch.compile) path.
//
// Reference counterparts: StickBreakingAttention (stickbreaking_attention/sb_varlen/__init__.py:23-67,
// sb_attn/__init__.py:15-53), varlen_fwd / varlen_bwd (sb_varlen/sb_varlen_fwd.py:411-452, sb_varlen_bwd.py:483-539).
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <cstdlib>
#include <mutex>

#include "../../include/sbattn.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// a negative SBATTN_E* code; becomes _lib.SbAttnError in Python
struct SbError : std::runtime_error {
    int code;
    std::string where;
    SbError(int c, const char* w) : std::runtime_error(std::string(w) + ": " + sbattn_strerror(c) + " (code " + std::to_string(c) + ")"), code(c), where(w) {}
};
void check(int rc, const char* where) {
    if (rc != 0) throw SbError(rc, where);
}

// one int32 word per device that the kernels OR their SBATTN_ST_* bits into; lives as long as the process (never freed: the
// CUDA context may be gone when static objects are destroyed)
Tensor status_word(int device) {
    static std::mutex mu;
    static auto* words = new std::vector<Tensor>();
    std::lock_guard<std::mutex> lock(mu);
    if ((int)words->size() <= device) words->resize(device + 1);
    Tensor& w = (*words)[device];
    if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
    return w;
}
uint32_t* status_ptr(int device) {
    static std::atomic<uint32_t*> ptr[64] = {};
    if (device >= 64) return (uint32_t*)status_word(device).data_ptr();
    uint32_t* p = ptr[device].load(std::memory_order_acquire);
    if (!p) {
        p = (uint32_t*)status_word(device).data_ptr();
        ptr[device].store(p, std::memory_order_release);
    }
    return p;
}
// SBATTN_CHECK_STATUS=1: every call synchronises and raises what the kernels reported
void maybe_check_status(int device) {
    const char* e = std::getenv("SBATTN_CHECK_STATUS");
    if (!e || e[0] != '1' || e[1] != 0) return;
    Tensor w = status_word(device);
    const int v = w.item<int>();
    w.zero_();
    TORCH_CHECK_VALUE(!(v & SBATTN_ST_BAD_SEQLENS), "cu_seqlens rejected on the device: ends must be non-decreasing, at most the number of "
                      "tokens, and no sequence longer than max_seqlens");
    TORCH_CHECK(!(v & SBATTN_ST_TIMEOUT), "a stick-breaking attention kernel gave up waiting (results are invalid)");
}

int dtype_of(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kBFloat16: return SBATTN_BF16;
        case at::kHalf: return SBATTN_F16;
        case at::kFloat: return SBATTN_F32;
        default: TORCH_CHECK_TYPE(false, "unsupported dtype ", t.scalar_type());
    }
}

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, int ndim) {
    TORCH_CHECK_VALUE(q.dim() == ndim && k.sizes() == q.sizes() && v.sizes() == q.sizes(), "q, k, v must share one ", ndim,
                      "-d shape, got ", q.sizes(), " ", k.sizes(), " ", v.sizes());
    TORCH_CHECK_TYPE(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), "q, k, v must share one dtype");
    TORCH_CHECK_VALUE(k.device() == q.device() && v.device() == q.device(), "q, k, v must live on one device");
    TORCH_CHECK_VALUE(q.size(-1) <= 128, "head_dim above 128 is not supported");
}
// Forward-mode differentiation is not implemented.  Refused here, for calls whose inputs need no gradient too: these pass the autograd
// node by, which would refuse it, and would drop the tangents without a word.
void refuse_forward_mode(const Tensor& q, const Tensor& k, const Tensor& v) {
    TORCH_CHECK_NOT_IMPLEMENTED(!q._fw_grad(0).defined() && !k._fw_grad(0).defined() && !v._fw_grad(0).defined(),
                                "stick-breaking attention does not implement forward mode AD");
}
void require_cuda(const Tensor& t) {
    TORCH_CHECK(t.is_cuda(), "stick-breaking attention runs on CUDA tensors only (there is no CPU implementation)");
}

// (cu_seqlens[0], longest sequence) of cumulative ends; `leading`: the first entry is the leading zero, not an end.  On a GPU one small
// kernel writes both to pinned memory and the host waits for its last word, not for a copy and the stream (us a call, 8 heads, 2048
// tokens in 6 documents, nothing but cu_seqlens given: forward 31 -> 25, forward and backward 110 -> 100).  When the stream has
// much to do before, waiting goes over to a stream synchronisation.
std::pair<int64_t, int64_t> seq_bounds(const Tensor& cu, bool leading, bool want_longest) {
    const Tensor c = cu.contiguous();
    const int64_t n = want_longest ? c.numel() : 1;
    if (c.is_cuda()) {
        c10::cuda::CUDAGuard guard(c.device());
        const auto st = c10::cuda::getCurrentCUDAStream();
        const Tensor host = at::empty({3}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
        volatile int64_t* out = host.data_ptr<int64_t>();
        out[2] = 0;
        check(sbattn_seq_bounds(c.const_data_ptr(), (int)c.element_size(), n, leading, (int64_t*)out, st.stream()), "sbattn_seq_bounds");
        for (int polls = 1; out[2] == 0; ++polls) {
            if (polls % 1024 != 0) continue;
            const cudaError_t e = polls < 64 * 1024 ? cudaStreamQuery(st) : cudaStreamSynchronize(st);
            if (e == cudaSuccess) break;  // the kernel is done, its writes are visible
            if (e != cudaErrorNotReady) C10_CUDA_CHECK(e);
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        return {out[0], out[1]};
    }
    const bool wide = c.scalar_type() == at::kLong;
    const auto at_ = [&](int64_t i) { return wide ? c.const_data_ptr<int64_t>()[i] : (int64_t)c.const_data_ptr<int32_t>()[i]; };
    int64_t longest = 0;
    for (int64_t i = leading ? 1 : 0; i < n; ++i) {
        const int64_t d = at_(i) - (i > 0 ? at_(i - 1) : 0);
        longest = i == (leading ? 1 : 0) ? d : std::max(longest, d);
    }
    return {at_(0), longest};
}

Tensor prep_cu(const Tensor& cu, const Tensor& q, std::optional<int64_t>& max_seqlens) {
    TORCH_CHECK_TYPE(cu.scalar_type() == at::kInt || cu.scalar_type() == at::kLong, "cu_seqlens must be int32 or int64");
    TORCH_CHECK_VALUE(cu.dim() == 1, "cu_seqlens must be 1-d");
    if (!max_seqlens) max_seqlens = cu.numel() == 0 ? 0 : seq_bounds(cu, false, true).second;
    Tensor c = cu.device() == q.device() ? cu : cu.to(q.device());
    return c.contiguous();
}

Tensor unit_inner(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
// Allocations past the dispatcher (~0.5 us each less): the caching allocator's memory all the same.  Not where torch fills new memory
// (torch.use_deterministic_algorithms): the rows of o behind the last sequence stay as they were allocated.
bool fills_memory() { return at::globalContext().deterministicAlgorithms() && at::globalContext().deterministicFillUninitializedMemory(); }
Tensor empty_like_dtype(const Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype) {
    return fills_memory() ? at::empty(sizes, t.options().dtype(dtype)) : at::detail::empty_cuda(sizes, dtype, t.device(), std::nullopt);
}
Tensor empty_rows(const Tensor& t) {
    if (t.is_non_overlapping_and_dense() && t.stride(-1) == 1)
        return fills_memory() ? at::empty_strided(t.sizes(), t.strides(), t.options())
                              : at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device());
    Tensor out = at::empty_like(t);
    return out.stride(-1) == 1 ? out : at::empty(t.sizes(), t.options());
}

SbMat mat(const Tensor& t, bool batched) {
    if (batched) return SbMat{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
    return SbMat{t.data_ptr(), 0, t.stride(0), t.stride(1)};
}
SbVec vec(const Tensor& t, bool batched) {
    if (batched) return SbVec{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
    return SbVec{t.data_ptr(), 0, t.stride(0), t.stride(1)};
}

// What describes a call besides its tensors
struct Opts {
    bool batched;
    int64_t max_seqlens;
    double scale;
    bool attend_current, fused;
    int path;
    bool f32_fused = false;  // out = o + rem * v in the kernels of float32 precision
};

SbParams base_params(const Tensor& q, const Tensor& cu, const Opts& o, bool save) {
    SbParams p{};
    p.dtype = dtype_of(q);
    p.path = o.path;
    if (o.batched) {
        p.batch = (int32_t)q.size(0);
        p.cu_width = 4;
        p.max_seqlen = (int32_t)q.size(2);
    } else {
        p.num_seqs = (int32_t)cu.numel();
        p.cu_width = (int32_t)cu.element_size();
        p.cu_seqlens = cu.data_ptr();
        p.max_seqlen = (int32_t)o.max_seqlens;
    }
    p.heads = (int32_t)q.size(-3);
    p.tokens = (int32_t)q.size(-2);
    p.head_dim = (int32_t)q.size(-1);
    p.attend_current = o.attend_current;
    p.inv_temp = (float)o.scale;
    p.save_carries = save;
    p.flags = o.fused ? SBATTN_FLAG_FUSED_REMAINDER : o.f32_fused ? SBATTN_FLAG_REMAINDER_IN_DV : 0;
    p.status = status_ptr(q.get_device());
    p.stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();
    return p;
}

Tensor bytes(size_t n, const Tensor& like) { return empty_like_dtype(like, {(int64_t)n}, at::kByte); }

struct FwdOut {
    Tensor o, rem, nla, ws;
};
// want_nla: the caller reads neg_log_acc.  It is a tensor of its own then, and where the workspace is kept for the backward (it would be
// kept with it); otherwise it lies behind the workspace, one allocation less, and goes with it.
FwdOut forward(Tensor q, Tensor k, Tensor v, const Tensor& cu, const Opts& opt, bool save, bool want_nla) {
    require_cuda(q);
    c10::cuda::OptionalCUDAGuard guard(q.device());
    q = unit_inner(q);
    k = unit_inner(k);
    v = unit_inner(v);
    FwdOut out;
    out.o = empty_rows(q);
    const auto rows = q.sizes().slice(0, q.dim() - 1);
    // no zero-fill: the library writes every row of rem and neg_log_acc
    out.rem = empty_like_dtype(q, rows, q.scalar_type());
    const bool own_nla = want_nla || save;
    if (own_nla) out.nla = empty_like_dtype(q, rows, at::kFloat);
    SbParams p = base_params(q, cu, opt, save);
    size_t fb = 0;
    check(sbattn_workspace_bytes(&p, &fb, nullptr), "sbattn_workspace_bytes");
    out.ws = bytes(fb + (own_nla ? 0 : 4 * (size_t)out.rem.numel()), q);  // fb is a multiple of 4
    p.q = mat(q, opt.batched);
    p.k = mat(k, opt.batched);
    p.v = mat(v, opt.batched);
    p.o = mat(out.o, opt.batched);
    p.rem = vec(out.rem, opt.batched);
    if (own_nla) {
        p.neg_log_acc = vec(out.nla, opt.batched);
    } else {
        p.neg_log_acc = vec(out.rem, opt.batched);  // same shape, contiguous as well
        p.neg_log_acc.ptr = (char*)out.ws.data_ptr() + fb;
    }
    p.fwd_workspace = out.ws.data_ptr();
    p.fwd_workspace_bytes = fb;
    check(sbattn_fwd(&p), "sbattn_fwd");
    maybe_check_status(q.get_device());
    return out;
}

bool tma_ok(const Tensor& t) {
    if (t.stride(-1) != 1 || ((uintptr_t)t.data_ptr() & 15)) return false;
    for (int64_t i = 0; i + 1 < t.dim(); ++i)
        if (t.stride(i) % 8 || (t.stride(i) < t.size(-1) && t.size(i) != 1)) return false;
    return true;
}

// a type and a head dim of the tensor-core kernels
bool tensor_type(const Tensor& q, int path) {
    const int64_t d = q.size(-1);
    return (q.scalar_type() == at::kBFloat16 || q.scalar_type() == at::kHalf) && (d == 32 || d == 64 || d == 128) && path != SBATTN_PATH_SIMT;
}
bool fusable(const Tensor& q, const Tensor& k, const Tensor& v, int path) {
    return tensor_type(q, path) && tma_ok(q) && tma_ok(k) && tma_ok(v);
}

std::array<Tensor, 3> backward(Tensor d_o, Tensor d_rem, Tensor q, Tensor k, Tensor v, const Tensor& cu, const Tensor& ws,
                               const Tensor& rem, const Opts& opt, int phases, const std::vector<Tensor>& out, const OptTensor& bwd_ws) {
    require_cuda(q);
    require_cuda(d_o);
    require_cuda(d_rem);
    require_cuda(ws);
    c10::cuda::OptionalCUDAGuard guard(q.device());
    q = unit_inner(q);
    k = unit_inner(k);
    v = unit_inner(v);
    d_o = unit_inner(d_o);
    if (d_o.scalar_type() != q.scalar_type()) d_o = d_o.to(q.scalar_type());
    // the fused backward exists in the tensor-core kernels only: give them an aligned copy
    if (opt.fused && !tma_ok(d_o)) d_o = d_o.contiguous().clone();
    if (d_rem.scalar_type() != q.scalar_type()) d_rem = d_rem.to(q.scalar_type());
    std::array<Tensor, 3> g;
    if (out.size() == 3) {
        g = {out[0], out[1], out[2]};
    } else {
        // no zero-fill: the library writes every row (rows outside all sequences included)
        g = {empty_rows(q), empty_rows(k), empty_rows(v)};
    }
    SbParams p = base_params(q, cu, opt, true);
    p.bwd_phases = phases;
    if (opt.f32_fused) d_rem = d_rem + (d_o * v).sum(-1);  // as autograd of o + rem * v forms it
    size_t fb = 0, bb = 0;
    check(sbattn_workspace_bytes(&p, &fb, &bb), "sbattn_workspace_bytes");
    TORCH_CHECK_VALUE((size_t)ws.numel() >= fb, "the forward workspace does not belong to this problem (was the forward run with no_grad?)");
    const Tensor bws = bwd_ws ? *bwd_ws : bytes(bb, q);
    TORCH_CHECK_VALUE((size_t)bws.numel() >= bb, "the backward workspace is too small");
    p.q = mat(q, opt.batched);
    p.k = mat(k, opt.batched);
    p.v = mat(v, opt.batched);
    p.d_o = mat(d_o, opt.batched);
    p.d_rem = vec(d_rem, opt.batched);
    if (opt.fused || opt.f32_fused) p.rem = vec(rem, opt.batched);
    p.dq = mat(g[0], opt.batched);
    p.dk = mat(g[1], opt.batched);
    p.dv = mat(g[2], opt.batched);
    p.fwd_workspace = ws.data_ptr();
    p.fwd_workspace_bytes = (size_t)ws.numel();
    p.bwd_workspace = bws.data_ptr();
    p.bwd_workspace_bytes = (size_t)bws.numel();
    check(sbattn_bwd(&p), "sbattn_bwd");
    maybe_check_status(q.get_device());
    return g;
}

// The autograd node.  `recompute`: nothing but the inputs and rem is kept, the backward runs the forward again for its carries.
struct StickBreaking : public torch::autograd::Function<StickBreaking> {
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                                                  const OptTensor& cu_seqlens, bool batched, int64_t max_seqlens, double scale, bool attend_current,
                                                  bool fused, bool recompute, int64_t path, bool f32_fused) {
        const Opts opt{batched, max_seqlens, scale, attend_current, fused, (int)path, f32_fused};
        const Tensor cu = cu_seqlens.value_or(Tensor());
        FwdOut r = ::forward(q, k, v, cu, opt, !recompute, false);
        ctx->save_for_backward({q, k, v, cu, recompute ? Tensor() : r.ws, r.rem});
        ctx->saved_data["o"] = c10::ivalue::Tuple::create({batched, max_seqlens, scale, attend_current, fused, recompute, path, f32_fused});
        return {r.o, r.rem};
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const auto tuple = ctx->saved_data["o"].toTuple();
        const auto& e = tuple->elements();
        const Opts opt{e[0].toBool(), e[1].toInt(), e[2].toDouble(), e[3].toBool(), e[4].toBool(), (int)e[6].toInt(), e[7].toBool()};
        const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &cu = saved[3];
        const Tensor ws = e[5].toBool() ? ::forward(q, k, v, cu, opt, true, false).ws : saved[4];
        const auto g = ::backward(grads[0], grads[1], q, k, v, cu, ws, saved[5], opt, 0, {}, std::nullopt);
        Tensor none;
        return {g[0], g[1], g[2], none, none, none, none, none, none, none, none, none};
    }
};

// sb_attn_varlen (cu given) / sb_attn: (o, rem), differentiable
std::pair<Tensor, Tensor> attend(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& cu_seqlens, std::optional<int64_t> max_seqlens,
                                 double scale, bool attend_current, bool fused, bool recompute, int path) {
    const bool batched = !cu_seqlens.has_value();
    check_qkv(q, k, v, batched ? 4 : 3);
    refuse_forward_mode(q, k, v);
    Tensor cu;
    if (batched) max_seqlens = q.size(2);
    else cu = prep_cu(*cu_seqlens, q, max_seqlens);
    // Operands that could go to the tensor-core kernels but for their strides: the sum is formed here.  (Formed here it costs ten small
    // operations of autograd: forward and backward of 4 heads, 512 float32 tokens 135 -> 96 us with the sum in the kernels.)
    const bool other = fused && !fusable(q, k, v, path), f32_fused = other && !tensor_type(q, path), compose = other && !f32_fused;
    if (other) fused = false;
    const auto done = [&](const Tensor& o, const Tensor& rem) {
        return std::pair<Tensor, Tensor>{compose ? o + rem.unsqueeze(-1) * v : o, rem};
    };
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
        require_cuda(q);
        auto r = StickBreaking::apply(q, k, v, batched ? OptTensor() : OptTensor(cu), batched, *max_seqlens, scale, attend_current, fused, recompute, (int64_t)path, f32_fused);
        return done(r[0], r[1]);
    }
    FwdOut r = forward(q, k, v, cu, Opts{batched, *max_seqlens, scale, attend_current, fused, path, f32_fused}, false, false);
    return done(r.o, r.rem);
}

// varlen_fwd / attn_fwd: (o, rem, neg_log_acc, workspace)
std::tuple<Tensor, Tensor, Tensor, Tensor> fwd(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& cu_seqlens,
                                               std::optional<int64_t> max_seqlens, double scale, bool attend_current, bool no_grad, bool fused,
                                               int path) {
    at::NoGradGuard guard;
    const bool batched = !cu_seqlens.has_value();
    check_qkv(q, k, v, batched ? 4 : 3);
    Tensor cu;
    if (batched) max_seqlens = q.size(2);
    else cu = prep_cu(*cu_seqlens, q, max_seqlens);
    FwdOut r = forward(q, k, v, cu, Opts{batched, *max_seqlens, scale, attend_current, fused, path}, !no_grad, true);
    return {r.o, r.rem, r.nla, r.ws};
}
// varlen_bwd / attn_bwd: (dq, dk, dv)
std::array<Tensor, 3> bwd(const Tensor& d_o, const Tensor& d_rem, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& cu_seqlens,
                          std::optional<int64_t> max_seqlens, const Tensor& ws, double scale, bool attend_current, int phases, bool fused,
                          const OptTensor& rem, int path, const std::vector<Tensor>& out, const OptTensor& bwd_ws) {
    at::NoGradGuard guard;
    const bool batched = !cu_seqlens.has_value();
    check_qkv(q, k, v, batched ? 4 : 3);
    TORCH_CHECK_VALUE(!fused || (rem && rem->sizes() == q.sizes().slice(0, q.dim() - 1) && rem->scalar_type() == q.scalar_type() && rem->device() == q.device()),
                      "the backward of the fused sum needs the forward's rem: the leading sizes, dtype and device of q");
    Tensor cu;
    if (batched) max_seqlens = q.size(2);
    else cu = prep_cu(*cu_seqlens, q, max_seqlens);
    return backward(d_o, d_rem, q, k, v, cu, ws, rem ? *rem : Tensor(), Opts{batched, *max_seqlens, scale, attend_current, fused, path}, phases, out, bwd_ws);
}

}  // namespace

PYBIND11_MODULE(_binding, m) {
    m.doc() = "Native host path of stickbreaking_attention_b200 (see csrc/sb_torch.cpp)";
    m.attr("built_for") = SBATTN_BUILT_FOR;  // read by build.py
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const SbError& e) {
            py::object cls = py::module_::import("stickbreaking_attention_b200._lib").attr("SbAttnError");
            PyErr_SetObject(cls.ptr(), cls(e.code, e.where).ptr());
        } catch (const py::builtin_exception&) {
            throw;
        } catch (const py::error_already_set&) {
            throw;
        } catch (...) {  // torch's exceptions with their Python types (ValueError, TypeError, RuntimeError)
            torch::translate_exception_to_python(p);
        }
    });
    // Without the interpreter lock: the calls may wait for the GPU (seq_bounds does, an allocation and the status check may), and what the
    // GPU has queued may in turn wait for another Python thread.
    const auto unlocked = py::call_guard<py::gil_scoped_release>();
    m.def("attend", &attend, unlocked);
    m.def("fwd", &fwd, unlocked);
    m.def("bwd", &bwd, unlocked);
    m.def("seq_bounds", &seq_bounds, unlocked);
    m.def("status_word", &status_word, unlocked);
}

// The parts of the operator surface that need libtorch's C++ API: the autograd formulas of the six
// reference operators (their CUDA kernels are registered through the stable ABI, torch_shim.cpp) and
// this package's own operators mmq_multi, swiglu and lm_head_loss with theirs.
//
// Why not in Python: a formula registered there costs a call into the interpreter for every operator
// call, some 5 us without and 50 us with a gradient, against 8 to 60 us of kernel in a decode step or a
// dense projection.  Formulas (reference: torch_ggml_ops/mmq.py:19-80, grouped_mmq.py:60-250): only the
// packed weights and the routing are saved, only the activation gets a gradient, the input-gradient
// operators refuse a second derivative.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <algorithm>
#include <cmath>

#include "../../include/tgo_mmq.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::tensor_list;
using torch::autograd::Variable;
using torch::autograd::variable_list;

template <typename Fn>
const c10::TypedOperatorHandle<Fn> op(const char* name) {
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Fn>();
}
// the last dimension as a plain integer (a traced shape is specialised on it, as an int argument is)
int64_t last_size(const Tensor& t, int64_t dim) { return t.sym_size(dim).guard_int(__FILE__, __LINE__); }

Tensor call_mmq(const Tensor& x, const Tensor& w, int64_t qt, int64_t n) {
    static const auto h = op<Tensor(const Tensor&, const Tensor&, int64_t, int64_t)>("torch_ggml_ops::mmq");
    return h.call(x, w, qt, n);
}
Tensor call_mmq_dx(const Tensor& dy, const Tensor& w, int64_t qt, int64_t k) {
    static const auto h = op<Tensor(const Tensor&, const Tensor&, int64_t, int64_t)>("torch_ggml_ops::mmq_grad_input");
    return h.call(dy, w, qt, k);
}
Tensor call_grouped(const Tensor& x, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t n) {
    static const auto h =
        op<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t)>("torch_ggml_ops::grouped_mmq");
    return h.call(x, w, ei, eo, qt, n);
}
Tensor call_grouped_dx(const Tensor& dy, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t k) {
    static const auto h =
        op<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t)>("torch_ggml_ops::grouped_mmq_grad_input");
    return h.call(dy, w, ei, eo, qt, k);
}
std::tuple<Tensor, Tensor> call_pair(const Tensor& x, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t n) {
    static const auto h = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t)>(
        "torch_ggml_ops::grouped_mmq_pair");
    return h.call(x, w0, w1, ei, eo, qt, n);
}
Tensor call_pair_dx(const Tensor& d0, const Tensor& d1, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t k) {
    static const auto h = op<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t)>(
        "torch_ggml_ops::grouped_mmq_pair_grad_input");
    return h.call(d0, d1, w0, w1, ei, eo, qt, k);
}

bool wants_grad(const Tensor& t) { return at::GradMode::is_enabled() && t.requires_grad(); }
// A cotangent handed over by autograd may be a transposed view; the operators refuse what is not
// contiguous.  (One that starts inside a storage stays as it is, and is refused.)
Tensor plain(const Tensor& g) { return g.contiguous(); }

[[noreturn]] void no_second_order(const char* name) {
    TORCH_CHECK(false, "torch_ggml_ops::", name, " does not support higher-order gradients");
}

// ------------------------------------------------------------------ dense
struct MmqFn : public Function<MmqFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, int64_t qt, int64_t n) {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->save_for_backward({w});
        ctx->saved_data["qt"] = qt;
        ctx->saved_data["k"] = last_size(x, -1);
        return call_mmq(x, w, qt, n);
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        Tensor dx;
        if (ctx->needs_input_grad(0) && g[0].defined())
            dx = call_mmq_dx(plain(g[0]), ctx->get_saved_variables()[0], ctx->saved_data["qt"].toInt(), ctx->saved_data["k"].toInt());
        return {dx, Tensor(), Tensor(), Tensor()};
    }
};
Tensor mmq_autograd(const Tensor& x, const Tensor& w, int64_t qt, int64_t n) {
    if (wants_grad(x)) return MmqFn::apply(x, w, qt, n);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_mmq(x, w, qt, n);
}

struct MmqDxFn : public Function<MmqDxFn> {
    static Tensor forward(AutogradContext*, const Tensor& dy, const Tensor& w, int64_t qt, int64_t k) {
        at::AutoDispatchBelowADInplaceOrView guard;
        return call_mmq_dx(dy, w, qt, k);
    }
    static tensor_list backward(AutogradContext*, tensor_list) { no_second_order("mmq_grad_input"); }
};
Tensor mmq_dx_autograd(const Tensor& dy, const Tensor& w, int64_t qt, int64_t k) {
    if (wants_grad(dy)) return MmqDxFn::apply(dy, w, qt, k);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_mmq_dx(dy, w, qt, k);
}

// ------------------------------------------------------------------ grouped
struct GroupedFn : public Function<GroupedFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t n) {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->save_for_backward({w, ei, eo});
        ctx->saved_data["qt"] = qt;
        ctx->saved_data["k"] = last_size(x, 1);
        return call_grouped(x, w, ei, eo, qt, n);
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        Tensor dx;
        if (ctx->needs_input_grad(0) && g[0].defined()) {
            const variable_list s = ctx->get_saved_variables();
            dx = call_grouped_dx(plain(g[0]), s[0], s[1], s[2], ctx->saved_data["qt"].toInt(), ctx->saved_data["k"].toInt());
        }
        return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
Tensor grouped_autograd(const Tensor& x, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t n) {
    if (wants_grad(x)) return GroupedFn::apply(x, w, ei, eo, qt, n);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_grouped(x, w, ei, eo, qt, n);
}

struct GroupedDxFn : public Function<GroupedDxFn> {
    static Tensor forward(AutogradContext*, const Tensor& dy, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t k) {
        at::AutoDispatchBelowADInplaceOrView guard;
        return call_grouped_dx(dy, w, ei, eo, qt, k);
    }
    static tensor_list backward(AutogradContext*, tensor_list) { no_second_order("grouped_mmq_grad_input"); }
};
Tensor grouped_dx_autograd(const Tensor& dy, const Tensor& w, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t k) {
    if (wants_grad(dy)) return GroupedDxFn::apply(dy, w, ei, eo, qt, k);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_grouped_dx(dy, w, ei, eo, qt, k);
}

// ------------------------------------------------------------------ pair
struct PairFn : public Function<PairFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo,
                                 int64_t qt, int64_t n) {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->save_for_backward({w0, w1, ei, eo});
        ctx->saved_data["qt"] = qt;
        ctx->saved_data["k"] = last_size(x, 1);
        ctx->set_materialize_grads(false);   // an unused projection has no cotangent
        auto [y0, y1] = call_pair(x, w0, w1, ei, eo, qt, n);
        return {y0, y1};
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        Tensor dx;
        if (ctx->needs_input_grad(0)) {
            const variable_list s = ctx->get_saved_variables();
            const int64_t qt = ctx->saved_data["qt"].toInt(), k = ctx->saved_data["k"].toInt();
            // both cotangents: the two products are summed in fp32 before one rounding
            if (g[0].defined() && g[1].defined()) dx = call_pair_dx(plain(g[0]), plain(g[1]), s[0], s[1], s[2], s[3], qt, k);
            else if (g[0].defined()) dx = call_grouped_dx(plain(g[0]), s[0], s[2], s[3], qt, k);
            else if (g[1].defined()) dx = call_grouped_dx(plain(g[1]), s[1], s[2], s[3], qt, k);
        }
        return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
std::tuple<Tensor, Tensor> pair_autograd(const Tensor& x, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t n) {
    if (wants_grad(x)) {
        const variable_list y = PairFn::apply(x, w0, w1, ei, eo, qt, n);
        return {y[0], y[1]};
    }
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_pair(x, w0, w1, ei, eo, qt, n);
}

struct PairDxFn : public Function<PairDxFn> {
    static Tensor forward(AutogradContext*, const Tensor& d0, const Tensor& d1, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo,
                          int64_t qt, int64_t k) {
        at::AutoDispatchBelowADInplaceOrView guard;
        return call_pair_dx(d0, d1, w0, w1, ei, eo, qt, k);
    }
    static tensor_list backward(AutogradContext*, tensor_list) { no_second_order("grouped_mmq_pair_grad_input"); }
};
Tensor pair_dx_autograd(const Tensor& d0, const Tensor& d1, const Tensor& w0, const Tensor& w1, const Tensor& ei, const Tensor& eo, int64_t qt, int64_t k) {
    if (wants_grad(d0) || wants_grad(d1)) return PairDxFn::apply(d0, d1, w0, w1, ei, eo, qt, k);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_pair_dx(d0, d1, w0, w1, ei, eo, qt, k);
}

// ------------------------------------------------------------------ mmq_multi
void check_rc(int rc, const char* what) { TORCH_CHECK(rc == TGO_OK, what, " failed: ", tgo_last_error()); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

void check_activation(const Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.storage_offset() == 0, name,
                " must be a contiguous torch.bfloat16 tensor with zero storage offset; torch_ggml_ops will not insert a hidden copy");
    TORCH_CHECK(t.dim() >= 1, name, " must have at least one dimension");
}
int64_t block_bytes(int64_t qt) {
    const int64_t b = qt >= 0 && qt <= INT32_MAX ? tgo_block_bytes(static_cast<int>(qt)) : -1;
    TORCH_CHECK(b > 0, "unsupported quant_type: ", qt);
    return b;
}

std::vector<Tensor> multi_cuda(const Tensor& x, at::TensorList ws, int64_t qt, int64_t n) {
    TORCH_CHECK(ws.size() >= 1 && ws.size() <= 4, "mmq_multi takes 1 to 4 packed weights; got ", ws.size());
    check_activation(x, "input");
    const int64_t k = x.size(-1);
    TORCH_CHECK(k > 0 && k % 256 == 0, "in_features must be a positive multiple of 256; got ", k);
    const int64_t rows = x.numel() / k, expected = n * (k / 256) * block_bytes(qt);
    const void* wp[4];
    void* yp[4];
    std::vector<Tensor> ys;
    ys.reserve(ws.size());
    auto sizes = x.sizes().vec();
    sizes.back() = n;
    const c10::cuda::CUDAGuard guard(x.device());
    for (size_t i = 0; i < ws.size(); ++i) {
        const Tensor& w = ws[i];
        TORCH_CHECK(w.scalar_type() == at::kByte && w.is_contiguous() && w.numel() == expected && w.device() == x.device(),
                    "every packed_weight must be a contiguous torch.uint8 tensor of ", expected, " bytes on the input's device");
        wp[i] = w.const_data_ptr();
        ys.push_back(at::empty(sizes, x.options()));
        yp[i] = ys.back().mutable_data_ptr();
    }
    check_rc(tgo_mmq_fwd_multi(x.const_data_ptr(), wp, yp, static_cast<int64_t>(ws.size()), rows, n, k, static_cast<int>(qt), stream_of(x)),
             "tgo_mmq_fwd_multi");
    return ys;
}
// its integers may be symbolic in a traced program
std::vector<Tensor> call_multi(const Tensor& x, at::TensorList ws, c10::SymInt qt, c10::SymInt n) {
    static const auto h = op<std::vector<Tensor>(const Tensor&, at::TensorList, c10::SymInt, c10::SymInt)>("torch_ggml_ops_b200::mmq_multi");
    return h.call(x, ws, std::move(qt), std::move(n));
}
struct MultiFn : public Function<MultiFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, std::vector<Tensor> ws, c10::SymInt qt, c10::SymInt n) {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->saved_data["qt"] = qt.guard_int(__FILE__, __LINE__);
        ctx->saved_data["k"] = last_size(x, -1);
        ctx->set_materialize_grads(false);
        variable_list y = call_multi(x, ws, std::move(qt), std::move(n));
        ctx->save_for_backward(std::move(ws));
        return y;
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        Tensor total;
        if (ctx->needs_input_grad(0)) {
            const variable_list ws = ctx->get_saved_variables();
            const int64_t qt = ctx->saved_data["qt"].toInt(), k = ctx->saved_data["k"].toInt();
            for (size_t i = 0; i < ws.size(); ++i) {
                if (!g[i].defined()) continue;
                Tensor dx = call_mmq_dx(plain(g[i]), ws[i], qt, k);
                total = total.defined() ? total + dx : dx;
            }
        }
        return {total, Tensor(), Tensor(), Tensor()};
    }
};
std::vector<Tensor> multi_autograd(const Tensor& x, at::TensorList ws, c10::SymInt qt, c10::SymInt n) {
    if (wants_grad(x)) return MultiFn::apply(x, ws.vec(), std::move(qt), std::move(n));
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_multi(x, ws, std::move(qt), std::move(n));
}

// ------------------------------------------------------------------ swiglu
void check_gate_up(const Tensor& g, const Tensor& u) {
    TORCH_CHECK(g.sizes() == u.sizes() && g.scalar_type() == at::kBFloat16 && u.scalar_type() == at::kBFloat16,
                "gate and up must be torch.bfloat16 tensors of the same shape");
}
Tensor swiglu_cuda(const Tensor& gate, const Tensor& up) {
    check_gate_up(gate, up);
    TORCH_CHECK(gate.dim() >= 1 && gate.device() == up.device(), "gate and up must be on the same device");
    const Tensor g = gate.contiguous(), u = up.contiguous();
    Tensor out = at::empty_like(g);
    const int64_t width = g.size(-1);
    const c10::cuda::CUDAGuard guard(g.device());
    check_rc(tgo_swiglu_fwd(g.const_data_ptr(), u.const_data_ptr(), nullptr, out.mutable_data_ptr(), width > 0 ? g.numel() / width : 0, width,
                            nullptr, stream_of(g)),
             "tgo_swiglu_fwd");
    return out;
}
std::tuple<Tensor, Tensor> swiglu_grad_cuda(const Tensor& grad, const Tensor& gate, const Tensor& up) {
    check_gate_up(gate, up);
    TORCH_CHECK(grad.sizes() == gate.sizes() && grad.scalar_type() == at::kBFloat16 && grad.device() == gate.device() && gate.device() == up.device(),
                "grad must be a torch.bfloat16 tensor like gate and up");
    const Tensor d = grad.contiguous(), g = gate.contiguous(), u = up.contiguous();
    Tensor dg = at::empty_like(g), du = at::empty_like(g);
    const int64_t width = g.size(-1);
    const c10::cuda::CUDAGuard guard(g.device());
    check_rc(tgo_swiglu_bwd(d.const_data_ptr(), g.const_data_ptr(), u.const_data_ptr(), nullptr, dg.mutable_data_ptr(), du.mutable_data_ptr(),
                            width > 0 ? g.numel() / width : 0, width, nullptr, stream_of(g)),
             "tgo_swiglu_bwd");
    return {dg, du};
}
Tensor call_swiglu(const Tensor& g, const Tensor& u) {
    static const auto h = op<Tensor(const Tensor&, const Tensor&)>("torch_ggml_ops_b200::swiglu");
    return h.call(g, u);
}
struct SwigluFn : public Function<SwigluFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& g, const Tensor& u) {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->save_for_backward({g, u});
        return call_swiglu(g, u);
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list d) {
        static const auto h =
            op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&)>("torch_ggml_ops_b200::swiglu_grad");
        const variable_list s = ctx->get_saved_variables();
        auto [dg, du] = h.call(d[0], s[0], s[1]);
        return {dg, du};
    }
};
Tensor swiglu_autograd(const Tensor& g, const Tensor& u) {
    if (wants_grad(g) || wants_grad(u)) return SwigluFn::apply(g, u);
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_swiglu(g, u);
}
struct SwigluGradFn : public Function<SwigluGradFn> {
    static variable_list forward(AutogradContext*, const Tensor& d, const Tensor& g, const Tensor& u) {
        at::AutoDispatchBelowADInplaceOrView guard;
        static const auto h =
            op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&)>("torch_ggml_ops_b200::swiglu_grad");
        auto [dg, du] = h.call(d, g, u);
        return {dg, du};
    }
    static tensor_list backward(AutogradContext*, tensor_list) {
        TORCH_CHECK(false, "torch_ggml_ops_b200::swiglu_grad does not support higher-order gradients");
    }
};
std::tuple<Tensor, Tensor> swiglu_grad_autograd(const Tensor& d, const Tensor& g, const Tensor& u) {
    if (wants_grad(d) || wants_grad(g) || wants_grad(u)) {
        const variable_list r = SwigluGradFn::apply(d, g, u);
        return {r[0], r[1]};
    }
    at::AutoDispatchBelowADInplaceOrView guard;
    static const auto h = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&)>("torch_ggml_ops_b200::swiglu_grad");
    return h.call(d, g, u);
}

// ------------------------------------------------------------------ lm_head_loss
// loss, d_hidden and, if asked for, d_hidden before its rounding
std::tuple<Tensor, Tensor, Tensor> lm_head_run(const Tensor& hidden, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& targets,
                                               int64_t chunk_rows, double grad_scale, bool want_f32) {
    TORCH_CHECK(hidden.is_cuda(), "input must be a CUDA tensor");
    TORCH_CHECK(hidden.scalar_type() == at::kBFloat16, "input must have dtype torch.bfloat16");
    TORCH_CHECK(hidden.dim() == 2, "hidden must have shape [rows, in_features]");
    TORCH_CHECK(w.is_cuda() && w.device() == hidden.device(), "input and packed_weight must be on the same device");
    TORCH_CHECK(w.scalar_type() == at::kByte, "packed_weight must have dtype torch.uint8");
    TORCH_CHECK(w.is_contiguous(), "packed_weight must be contiguous; torch_ggml_ops will not insert a hidden copy");
    TORCH_CHECK(w.storage_offset() == 0, "packed_weight must have zero storage offset");
    TORCH_CHECK(targets.device() == hidden.device() && targets.scalar_type() == at::kLong && targets.is_contiguous(),
                "targets must be a contiguous torch.int64 tensor on the input's device");
    const int64_t rows = hidden.size(0), k = hidden.size(1);
    TORCH_CHECK(targets.numel() == rows, "targets must have one entry per row of hidden");
    TORCH_CHECK(k > 0 && k % 256 == 0, "input width must be a positive multiple of 256; got ", k);
    TORCH_CHECK(vocab > 0, "out_features must be positive; got ", vocab);
    const int64_t expected = vocab * (k / 256) * block_bytes(qt);
    TORCH_CHECK(w.numel() == expected, "packed_weight has ", w.numel(), " bytes, expected ", expected, " for [", vocab, ", ", k, "] quant_type=", qt);
    TORCH_CHECK(chunk_rows > 0, "chunk_rows must be positive");
    if (!hidden.is_contiguous() && rows > 0) {
        // a chunk is copied where it is a view, and a copy keeps the order of the strides: rows may lie apart, columns not
        const int64_t chunk = std::min(chunk_rows, rows), last = rows % chunk;
        for (const int64_t n : {chunk, last > 0 ? last : chunk})
            TORCH_CHECK(at::empty_like(hidden.narrow(0, 0, n), hidden.options().device(at::kMeta)).is_contiguous(),
                        "input must be contiguous; torch_ggml_ops will not insert a hidden copy");
    }
    const c10::cuda::CUDAGuard guard(hidden.device());
    Tensor x = hidden.contiguous();
    if (reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16 != 0) x = x.clone();
    Tensor like_hidden = at::empty_like(hidden);
    Tensor d_hidden = like_hidden.is_contiguous() ? like_hidden : at::empty({rows, k}, x.options());
    Tensor d_f32 = want_f32 ? at::empty({rows, k}, x.options().dtype(at::kFloat)) : Tensor();
    if (rows == 0) return {at::zeros({}, x.options().dtype(at::kFloat)), like_hidden, d_f32};
    Tensor loss = at::empty({}, x.options().dtype(at::kFloat));
    const int64_t bytes = tgo_lm_head_loss_workspace_bytes(rows, vocab, k, static_cast<int>(qt), chunk_rows);
    TORCH_CHECK(bytes >= 0, "unsupported sizes");
    Tensor ws = at::empty({bytes}, x.options().dtype(at::kByte));
    check_rc(tgo_lm_head_loss_f32(x.const_data_ptr(), w.const_data_ptr(), targets.const_data_ptr<int64_t>(), rows, vocab, k, static_cast<int>(qt),
                                  chunk_rows, static_cast<float>(grad_scale), loss.mutable_data_ptr<float>(), d_hidden.mutable_data_ptr(),
                                  want_f32 ? d_f32.mutable_data_ptr<float>() : nullptr, ws.mutable_data_ptr(), bytes, stream_of(x)),
             "lm_head_loss");
    if (!like_hidden.is_contiguous()) like_hidden.copy_(d_hidden);
    return {loss, like_hidden, d_f32};
}
std::tuple<Tensor, Tensor> lm_head_cuda(const Tensor& hidden, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& targets, int64_t chunk_rows,
                                        double grad_scale) {
    auto [loss, d, f] = lm_head_run(hidden, w, qt, vocab, targets, chunk_rows, grad_scale, false);
    return {loss, d};
}
std::tuple<Tensor, Tensor, Tensor> lm_head_f32_cuda(const Tensor& hidden, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& targets,
                                                    int64_t chunk_rows, double grad_scale) {
    return lm_head_run(hidden, w, qt, vocab, targets, chunk_rows, grad_scale, true);
}
std::tuple<Tensor, Tensor> call_lm_head(const Tensor& x, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& t, int64_t chunk, double scale) {
    static const auto h = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, int64_t, int64_t, const Tensor&, int64_t, double)>(
        "torch_ggml_ops_b200::lm_head_loss");
    return h.call(x, w, qt, vocab, t, chunk, scale);
}
std::tuple<Tensor, Tensor, Tensor> call_lm_head_f32(const Tensor& x, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& t, int64_t chunk,
                                                    double scale) {
    static const auto h = op<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, int64_t, int64_t, const Tensor&, int64_t, double)>(
        "torch_ggml_ops_b200::lm_head_loss_f32");
    return h.call(x, w, qt, vocab, t, chunk, scale);
}
[[noreturn]] void no_second_order_head() { TORCH_CHECK(false, "torch_ggml_ops_b200::lm_head_loss does not support higher-order gradients"); }
// d * g * scale, the gradient that autograd gets: d in fp32, so that the product is rounded once.  The loss is not linear in hidden and d has no graph, so
// a second derivative is refused; `edge` ties the result to hidden for that.
struct LmHeadGradFn : public Function<LmHeadGradFn> {
    static Tensor forward(AutogradContext*, const Tensor& edge, const Tensor& d, const Tensor& g, double scale) {
        at::AutoDispatchBelowADInplaceOrView guard;
        return (d * (g * scale)).to(edge.scalar_type());
    }
    static tensor_list backward(AutogradContext*, tensor_list) { no_second_order_head(); }
};
// The gradient of the loss is the one the call has computed, without its scale.  `edge`: an empty tensor
// whose history is hidden's (hidden itself is not kept, so it may be overwritten before the backward pass).
struct LmHeadFn : public Function<LmHeadFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& edge, const Tensor& w, int64_t qt, int64_t vocab,
                                 const Tensor& t, int64_t chunk, double scale) {
        at::AutoDispatchBelowADInplaceOrView guard;
        // a scale that could be divided out again without leaving bf16's range serves both
        const bool serves = std::abs(scale) >= 0x1p-40 && std::abs(scale) <= 0x1p40;
        auto [loss, d, unscaled] = call_lm_head_f32(x, w, qt, vocab, t, chunk, scale);
        if (!serves) unscaled = std::get<2>(call_lm_head_f32(x, w, qt, vocab, t, chunk, 1.0));
        ctx->save_for_backward({unscaled, edge});
        ctx->saved_data["scale"] = serves ? 1.0 / scale : 1.0;
        ctx->set_materialize_grads(false);
        return {loss, d};
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        Tensor dx;
        if (g[1].defined()) no_second_order_head();   // d is a derivative already
        if (ctx->needs_input_grad(0) && g[0].defined()) {
            const variable_list s = ctx->get_saved_variables();
            dx = LmHeadGradFn::apply(s[1], s[0], g[0], ctx->saved_data["scale"].toDouble());
        }
        return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
std::tuple<Tensor, Tensor> lm_head_autograd(const Tensor& x, const Tensor& w, int64_t qt, int64_t vocab, const Tensor& t, int64_t chunk, double scale) {
    if (wants_grad(x)) {
        TORCH_CHECK(x.dim() == 2, "hidden must have shape [rows, in_features]");
        const variable_list r = LmHeadFn::apply(x, x.narrow(0, 0, 0).clone(), w, qt, vocab, t, chunk, scale);
        return {r[0], r[1]};
    }
    at::AutoDispatchBelowADInplaceOrView guard;
    return call_lm_head(x, w, qt, vocab, t, chunk, scale);
}

}  // namespace

TORCH_LIBRARY_IMPL(torch_ggml_ops, Autograd, m) {
    m.impl("mmq", &mmq_autograd);
    m.impl("mmq_grad_input", &mmq_dx_autograd);
    m.impl("grouped_mmq", &grouped_autograd);
    m.impl("grouped_mmq_grad_input", &grouped_dx_autograd);
    m.impl("grouped_mmq_pair", &pair_autograd);
    m.impl("grouped_mmq_pair_grad_input", &pair_dx_autograd);
}

TORCH_LIBRARY_FRAGMENT(torch_ggml_ops_b200, m) {
    m.def("mmq_multi(Tensor input, Tensor[] packed_weights, SymInt quant_type, SymInt out_features) -> Tensor[]");
    m.def("swiglu(Tensor gate, Tensor up) -> Tensor");
    m.def("swiglu_grad(Tensor grad, Tensor gate, Tensor up) -> (Tensor, Tensor)");
    m.def(
        "lm_head_loss(Tensor hidden, Tensor packed_weight, int quant_type, int vocab, Tensor targets, int chunk_rows, float grad_scale) -> "
        "(Tensor, Tensor)");
    m.def(
        "lm_head_loss_f32(Tensor hidden, Tensor packed_weight, int quant_type, int vocab, Tensor targets, int chunk_rows, float grad_scale) -> "
        "(Tensor, Tensor, Tensor)");
}
TORCH_LIBRARY_IMPL(torch_ggml_ops_b200, CUDA, m) {
    m.impl("mmq_multi", &multi_cuda);
    m.impl("swiglu", &swiglu_cuda);
    m.impl("swiglu_grad", &swiglu_grad_cuda);
    m.impl("lm_head_loss", &lm_head_cuda);
    m.impl("lm_head_loss_f32", &lm_head_f32_cuda);
}
TORCH_LIBRARY_IMPL(torch_ggml_ops_b200, Autograd, m) {
    m.impl("mmq_multi", &multi_autograd);
    m.impl("swiglu", &swiglu_autograd);
    m.impl("swiglu_grad", &swiglu_grad_autograd);
    m.impl("lm_head_loss", &lm_head_autograd);
}

// Importing the module runs the registrations above; it exports nothing else.
extern "C" PyObject* PyInit__ext(void) {
    static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ext", nullptr, -1, nullptr};
    return PyModule_Create(&module);
}

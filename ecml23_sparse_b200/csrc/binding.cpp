// CPython binding of the hot entry points over torch tensors: argument checks, output and scratch allocation,
// the call into the C ABI (include/ffi_b200.h) and the autograd node, all in one native call per operation.
//
// Why native: the kernels of a small layer take 30 to 100 us per training step, and the same steps written in Python over
// ctypes (device context manager, stream lookup, 20-argument foreign call, Python autograd function) took 60 to 90 us per
// direction, more than the GPU's work; see ops.py for the measured figures.
//
// Nothing here computes; there is no CPU path.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>
#include <pybind11/stl.h>

#include <list>
#include <memory>
#include <mutex>
#include <optional>
#include <tuple>
#include <vector>

#include "ffi_b200.h"

// read from the file by build.py: a module built for another torch is stale
extern "C" __attribute__((used, visibility("default"))) const char ffi_binding_torch[] = "ffi-binding-torch=" FFI_TORCH_VERSION;

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// ---- scratch: one grown buffer per (device, stream) --------------------------------------------------------
// A call holds its buffer's lock while it launches (and releases it before it raises, which needs the GIL), so two
// threads that share a stream cannot interleave kernels that use the same scratch.  At most kMaxScratch streams keep one; the least recently used goes back to torch's allocator
// (which hands it out again in stream order, so kernels still queued on that stream are safe).
struct Scratch {
    int device;
    cudaStream_t stream;
    std::mutex mu;
    Tensor buf;
};
constexpr size_t kMaxScratch = 64;
std::mutex g_scratch_mu;
std::list<std::shared_ptr<Scratch>> g_scratch;  // most recently used first

std::shared_ptr<Scratch> scratch_for(int device, cudaStream_t stream) {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    for (auto it = g_scratch.begin(); it != g_scratch.end(); ++it)
        if ((*it)->device == device && (*it)->stream == stream) {
            if (it != g_scratch.begin()) g_scratch.splice(g_scratch.begin(), g_scratch, it);
            return g_scratch.front();
        }
    auto s = std::make_shared<Scratch>();
    s->device = device;
    s->stream = stream;
    g_scratch.push_front(s);
    if (g_scratch.size() > kMaxScratch) g_scratch.pop_back();
    return s;
}

// Locks the stream's buffer, makes it hold `bytes` at a 256-byte aligned address (grown, never shrunk) and runs f on it.
template <class F>
int with_scratch(const at::Device& dev, cudaStream_t stream, size_t bytes, F&& f) {
    const std::shared_ptr<Scratch> s = scratch_for(dev.index(), stream);
    std::lock_guard<std::mutex> lock(s->mu);
    if (bytes == 0) return f(nullptr, 0);
    if (!s->buf.defined() || static_cast<size_t>(s->buf.numel()) < bytes + 256)
        s->buf = at::empty({static_cast<int64_t>((bytes + 256) * 5 / 4 + 256)}, at::TensorOptions(at::kByte).device(dev));
    const uintptr_t p = reinterpret_cast<uintptr_t>(s->buf.data_ptr());
    const uintptr_t off = (256 - p % 256) % 256;
    return f(reinterpret_cast<void*>(p + off), s->buf.numel() - off);
}

void clear_scratch() {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    g_scratch.clear();
}

// ---- errors ------------------------------------------------------------------------------------------------
void check(int status) {
    if (status == FFI_OK) return;
    const std::string text = ffi_last_error();
    py::gil_scoped_acquire gil;
    py::object cls = py::module_::import("ecml23_sparse_b200._lib").attr("FFIError");
    py::object exc = cls(status, text);
    PyErr_SetObject(cls.ptr(), exc.ptr());
    throw py::error_already_set();
}

std::string shape_text(const Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + ")";
}

Tensor cuda_matrix(const char* name, const Tensor& t, bool float_only) {
    if (!t.is_cuda()) throw py::value_error(std::string(name) + " must be a CUDA tensor: this library has no CPU path");
    const auto st = t.scalar_type();
    if (st != at::kFloat && (float_only || st != at::kBFloat16))
        throw py::type_error(std::string(name) + " has dtype " + c10::toString(st) +
                             (float_only ? ", expected float32" : ", expected float32 or bfloat16"));
    if (t.dim() != 2) throw py::value_error(std::string(name) + " must have rank 2, got shape " + shape_text(t));
    return t.contiguous();
}

// units, fan_in >= 0: the table or the weights come as a layer's flat vector of that many connections.
Tensor flat_vector(const char* name, const Tensor& t, int64_t units, int64_t fan_in) {
    if (!t.is_cuda()) throw py::value_error(std::string(name) + " must be a CUDA tensor: this library has no CPU path");
    if (t.dim() != 1 || t.size(0) != units * fan_in)
        throw py::value_error(std::string(name) + " must be a vector of units * fan_in elements, got shape " + shape_text(t));
    return t.contiguous();
}

Tensor index_matrix(const Tensor& t) {
    if (!t.is_cuda()) throw py::value_error("lookup must be a CUDA tensor: this library has no CPU path");
    if (t.scalar_type() != at::kInt && t.scalar_type() != at::kUInt32)
        throw py::type_error(std::string("lookup has dtype ") + c10::toString(t.scalar_type()) + ", expected int32 or uint32");
    if (t.dim() != 2) throw py::value_error("lookup must have rank 2, got shape " + shape_text(t));
    return t.contiguous();  // values < 2^31 by the reference's contract: one entry point serves both types
}

struct Operands {
    Tensor x, idx, W;
    int dtype;
    int64_t B, N, L, K;
    const int32_t* idx_ptr() const { return static_cast<const int32_t*>(idx.const_data_ptr()); }
};

Operands operands(const Tensor& features, const Tensor& lookup, const Tensor& weights, bool transposed, int64_t units = -1,
                  int64_t fan_in = -1) {
    Operands o;
    const bool flat = units >= 0;
    o.x = cuda_matrix("features", features, false);
    o.W = flat ? flat_vector("weights", weights, units, fan_in) : cuda_matrix("weights", weights, false);
    if (o.x.scalar_type() != o.W.scalar_type())
        throw py::type_error(std::string("features (") + c10::toString(o.x.scalar_type()) + ") and weights (" +
                             c10::toString(o.W.scalar_type()) + ") must have the same dtype");
    o.dtype = o.x.scalar_type() == at::kBFloat16 ? FFI_BF16 : FFI_F32;
    if (flat && lookup.scalar_type() != at::kInt) throw py::type_error("the layer's table must be int32");
    o.idx = flat ? flat_vector("lookup", lookup, units, fan_in) : index_matrix(lookup);
    if (o.idx.sizes() != o.W.sizes())
        throw py::value_error("lookup " + shape_text(o.idx) + " and weights " + shape_text(o.W) + " must have equal shapes");
    o.B = o.x.size(transposed ? 1 : 0);
    o.N = o.x.size(transposed ? 0 : 1);
    o.L = flat ? units : o.W.size(0);
    o.K = flat ? fan_in : o.W.size(1);
    return o;
}

Tensor f32(at::IntArrayRef shape, const at::Device& dev) {
    return at::empty(shape, at::TensorOptions(at::kFloat).device(dev));
}

const float* opt_f32(const OptTensor& t) { return t && t->defined() ? t->const_data_ptr<float>() : nullptr; }

OptTensor checked_bias(const OptTensor& bias, int64_t L) {
    if (!bias || !bias->defined()) return std::nullopt;
    if (bias->dim() != 1 || bias->size(0) != L || bias->scalar_type() != at::kFloat || !bias->is_cuda())
        throw py::value_error("bias must be a float32 CUDA tensor of shape [L]");
    return bias->contiguous();
}

// ---- the operations ----------------------------------------------------------------------------------------
Tensor run_forward(const Operands& o, const OptTensor& bias_in, bool transposed) {
    const OptTensor bias = checked_bias(bias_in, o.L);
    const c10::cuda::CUDAGuard guard(o.x.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(o.x.device().index());
    Tensor out = f32({o.B, o.L}, o.x.device());
    check(with_scratch(o.x.device(), stream, ffi_forward_workspace_bytes(o.B, o.N, o.L, o.K, transposed, o.dtype),
                       [&](void* ws, size_t len) {
                           return ffi_forward(o.x.const_data_ptr(), o.idx_ptr(), o.W.const_data_ptr(), opt_f32(bias),
                                              out.data_ptr<float>(), o.B, o.N, o.L, o.K, transposed, o.dtype, ws, len, stream);
                       }));
    return out;
}

Tensor forward(const Tensor& features, const Tensor& lookup, const Tensor& weights, const OptTensor& bias, bool transposed) {
    return run_forward(operands(features, lookup, weights, transposed), bias, transposed);
}

std::tuple<OptTensor, OptTensor, OptTensor> run_backward(const Operands& o, const Tensor& out_grad, bool transposed,
                                                         uintptr_t plan_handle, bool want_x, bool want_w, bool want_b,
                                                         bool grad_is_transposed, const OptTensor& gx_out) {
    const Tensor g = cuda_matrix("out_grad", out_grad, true);
    if (grad_is_transposed) {
        if (g.size(0) != o.L || g.size(1) < o.B)
            throw py::value_error("transposed out_grad has shape " + shape_text(g) + ", expected [" + std::to_string(o.L) +
                                  ", >= " + std::to_string(o.B) + "]");
    } else if (g.size(0) != o.B || g.size(1) != o.L) {
        throw py::value_error("out_grad has shape " + shape_text(g) + ", expected (" + std::to_string(o.B) + ", " +
                              std::to_string(o.L) + ")");
    }
    const at::Device dev = o.x.device();
    const c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
    OptTensor gx, gw, gb;
    if (want_x) {
        if (gx_out && gx_out->defined()) {
            if (gx_out->scalar_type() != at::kFloat || !gx_out->is_contiguous() || gx_out->numel() != o.x.numel() ||
                gx_out->device() != dev)
                throw py::value_error("feature_grad_out must be a contiguous float32 tensor of features' size on its device");
            gx = gx_out->view(o.x.sizes());
        } else {
            gx = f32(o.x.sizes(), dev);
        }
    }
    if (want_w) gw = f32({o.L, o.K}, dev);
    if (want_b) gb = f32({o.L}, dev);
    const ffi_plan* plan = reinterpret_cast<const ffi_plan*>(plan_handle);
    float* gxp = gx ? gx->data_ptr<float>() : nullptr;
    float* gwp = gw ? gw->data_ptr<float>() : nullptr;
    float* gbp = gb ? gb->data_ptr<float>() : nullptr;
    const float* gp = g.const_data_ptr<float>();
    check(with_scratch(
        dev, stream, ffi_backward_workspace_bytes(plan, o.B, o.N, o.L, o.K, transposed, o.dtype, want_x, want_w || want_b),
        [&](void* ws, size_t len) {
            return grad_is_transposed
                       ? ffi_backward_from_transposed(o.x.const_data_ptr(), o.idx_ptr(), o.W.const_data_ptr(), gp, g.size(1), plan,
                                                      gxp, gwp, gbp, o.B, o.N, o.L, o.K, transposed, o.dtype, ws, len, stream)
                       : ffi_backward(o.x.const_data_ptr(), o.idx_ptr(), o.W.const_data_ptr(), gp, plan, gxp, gwp, gbp, o.B, o.N,
                                      o.L, o.K, transposed, o.dtype, ws, len, stream);
        }));
    return {gx, gw, gb};
}

std::tuple<OptTensor, OptTensor, OptTensor> backward(const Tensor& features, const Tensor& lookup, const Tensor& weights,
                                                     const Tensor& out_grad, bool transposed, uintptr_t plan_handle,
                                                     bool want_x, bool want_w, bool want_b, bool grad_is_transposed,
                                                     const OptTensor& gx_out) {
    return run_backward(operands(features, lookup, weights, transposed), out_grad, transposed, plan_handle, want_x, want_w,
                        want_b, grad_is_transposed, gx_out);
}

Tensor device_int32(const Tensor& t, const at::Device& dev) {
    return t.to(at::TensorOptions(at::kInt).device(dev)).contiguous();
}

std::tuple<Tensor, Tensor> forward_loss(int kind, const Tensor& features, const Tensor& lookup, const Tensor& weights,
                                        const OptTensor& bias_in, const Tensor& row_ptr_in, const Tensor& labels_in,
                                        bool transposed, int64_t total_labels, int64_t label_offset, const OptTensor& loss_out) {
    const Operands o = operands(features, lookup, weights, transposed);
    const at::Device dev = o.x.device();
    const c10::cuda::CUDAGuard guard(dev);
    const Tensor row_ptr = device_int32(row_ptr_in, dev), labels = device_int32(labels_in, dev);
    if (row_ptr.numel() != o.B + 1) throw py::value_error("row_ptr must have B+1 entries");
    Tensor loss;
    if (loss_out && loss_out->defined()) {
        if (loss_out->scalar_type() != at::kFloat || loss_out->numel() != 1 || loss_out->device() != dev)
            throw py::value_error("loss_out must be one fp32 element on the features' device");
        loss = *loss_out;
    } else {
        loss = f32({}, dev);
    }
    const int64_t ldg = ffi_transposed_gradient_stride(o.B);
    Tensor gT = f32({o.L, ldg}, dev);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
    const int32_t* rp = row_ptr.const_data_ptr<int32_t>();
    const int32_t* lp = labels.numel() ? labels.const_data_ptr<int32_t>() : rp;
    check(with_scratch(dev, stream, ffi_forward_bce_workspace_bytes(o.B, o.N, o.L, o.K, transposed, o.dtype),
                       [&](void* ws, size_t len) {
                           return ffi_forward_loss(kind, o.x.const_data_ptr(), o.idx_ptr(), o.W.const_data_ptr(),
                                                   opt_f32(bias_in), rp, lp, gT.data_ptr<float>(), loss.data_ptr<float>(), o.B,
                                                   o.N, o.L, o.K, total_labels > 0 ? total_labels : o.L, label_offset,
                                                   transposed, o.dtype, ws, len, stream);
                       }));
    return {loss, gT};
}

std::tuple<Tensor, Tensor> forward_topk(const Tensor& features, const Tensor& lookup, const Tensor& weights,
                                        const OptTensor& bias_in, int64_t k, bool transposed, int64_t label_offset) {
    const Operands o = operands(features, lookup, weights, transposed);
    const at::Device dev = o.x.device();
    const c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
    Tensor val = f32({o.B, k}, dev);
    Tensor lab = at::empty({o.B, k}, at::TensorOptions(at::kInt).device(dev));
    check(with_scratch(dev, stream, ffi_forward_topk_workspace_bytes(o.B, o.N, o.L, o.K, transposed, o.dtype),
                       [&](void* ws, size_t len) {
                           return ffi_forward_topk(o.x.const_data_ptr(), o.idx_ptr(), o.W.const_data_ptr(), opt_f32(bias_in),
                                                   val.data_ptr<float>(), lab.data_ptr<int32_t>(), static_cast<int>(k), o.B,
                                                   o.N, o.L, o.K, label_offset, transposed, o.dtype, ws, len, stream);
                       }));
    return {val, lab};
}

void adam_step(const std::vector<std::tuple<Tensor, Tensor, Tensor, Tensor>>& params, double lr, double beta1, double beta2,
               double eps, int64_t step) {
    std::vector<ffi_adam_tensor> group;
    std::vector<Tensor> held;  // contiguous copies live until the launch
    at::Device dev(at::kCUDA, 0);
    const auto flush = [&] {
        if (group.empty()) return;
        const c10::cuda::CUDAGuard guard(dev);
        check(ffi_adam_step_group(group.data(), static_cast<int>(group.size()), static_cast<float>(lr), static_cast<float>(beta1),
                                  static_cast<float>(beta2), static_cast<float>(eps), step,
                                  c10::cuda::getCurrentCUDAStream(dev.index())));
        group.clear();
    };
    for (const auto& [p, m, v, grad] : params) {
        const Tensor g = grad.contiguous();
        if (g.scalar_type() != at::kFloat || g.sizes() != p.sizes() || !g.is_cuda())
            throw py::value_error("gradient must be float32 with the parameter's shape");
        if (dev != p.device()) flush();
        dev = p.device();
        held.push_back(g);
        if (p.numel() > 0)
            group.push_back({p.data_ptr(), m.data_ptr<float>(), v.data_ptr<float>(), g.const_data_ptr<float>(), p.numel(),
                             p.scalar_type() == at::kBFloat16 ? FFI_BF16 : FFI_F32});
    }
    flush();
}

// ---- autograd (gradient registration of sparse/ops/fixed_fan_in_ops.py:31-40: [feature_grad, None, weight_grad]) ----

// The cached plan of a table; Python owns the cache (ops.get_plan), so that a plan keeps its table alive and an in-place
// update of the table leads to a rebuild.
py::object* g_get_plan = nullptr;

struct PlanRef {
    py::object plan;  // keeps the plan alive until the launches are queued
    uintptr_t handle = 0;
    PlanRef(const Tensor& lookup, int64_t n_in) {
        py::gil_scoped_acquire gil;
        plan = (*g_get_plan)(lookup, n_in);
        handle = plan.attr("address").cast<uintptr_t>();
    }
    ~PlanRef() {
        py::gil_scoped_acquire gil;
        plan = py::object();
    }
};

// `layer`: features come as [B,N] and are handed to the transposed op (sparse/custom_layer.py:45-50); the table and the
// weights are the layer's flat vectors.
struct FanInSparseMatmul : public torch::autograd::Function<FanInSparseMatmul> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& features, const Tensor& lookup,
                          const Tensor& weights, const OptTensor& bias, bool transposed, bool layer, int64_t units, int64_t fan_in) {
        const Tensor x = layer ? turned(features) : features;
        ctx->saved_data["flags"] = static_cast<int64_t>(transposed) | (layer ? 2 : 0) | (bias && bias->defined() ? 4 : 0);
        // of a layer x is this node's own transposed copy; table and weights are saved as the caller's tensors, so that an
        // in-place change between forward and backward is noticed
        ctx->save_for_backward({x, lookup, weights});
        return run_forward(operands(x, lookup, weights, transposed, layer ? units : -1, fan_in), bias, transposed);
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const int64_t flags = ctx->saved_data["flags"].toInt();
        const bool transposed = flags & 1, layer = flags & 2;
        const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(2);
        const bool need_b = (flags & 4) && ctx->needs_input_grad(3);
        const int64_t units = layer ? grads[0].size(1) : -1, fan_in = layer ? saved[2].numel() / units : -1;
        std::optional<PlanRef> plan;
        if (need_x) plan.emplace(layer ? saved[1].view({units, fan_in}) : saved[1], saved[0].size(transposed ? 0 : 1));
        auto [gx, gw, gb] = run_backward(operands(saved[0], saved[1], saved[2], transposed, units, fan_in), grads[0], transposed,
                                         plan ? plan->handle : 0, need_x, need_w, need_b, false, std::nullopt);
        torch::autograd::variable_list out(8);
        if (gx) out[0] = layer ? gx->t() : *gx;
        if (gw) out[2] = layer ? gw->view({-1}) : *gw;
        if (gb) out[3] = *gb;
        return out;
    }

    // [B,N] -> a contiguous [N,B] (sparse/custom_layer.py:48)
    static Tensor turned(const Tensor& x) {
        if (!x.is_cuda() || x.scalar_type() != at::kFloat || x.dim() != 2 || !x.is_contiguous() || x.numel() == 0)
            return x.t().contiguous();
        const c10::cuda::CUDAGuard guard(x.device());
        Tensor out = f32({x.size(1), x.size(0)}, x.device());
        check(ffi_transpose_features(x.const_data_ptr<float>(), out.data_ptr<float>(), x.size(0), x.size(1),
                                     c10::cuda::getCurrentCUDAStream(x.device().index())));
        return out;
    }
};

Tensor matmul(const Tensor& features, const Tensor& lookup, const Tensor& weights, const OptTensor& bias, bool transposed) {
    return FanInSparseMatmul::apply(features, lookup, weights, bias, transposed, false, int64_t(0), int64_t(0));
}

Tensor layer_forward(const Tensor& inputs, const Tensor& indices, const Tensor& weights, const OptTensor& bias, int64_t units,
                     int64_t fan_in) {
    return FanInSparseMatmul::apply(inputs, indices, weights, bias, true, true, units, fan_in);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using Unlocked = py::call_guard<py::gil_scoped_release>;  // other Python threads run while the kernels are launched
    m.def("forward", &forward, Unlocked());
    m.def("backward", &backward, Unlocked());
    m.def("forward_loss", &forward_loss, Unlocked());
    m.def("forward_topk", &forward_topk, Unlocked());
    m.def("adam_step", &adam_step, Unlocked());
    m.def("matmul", &matmul, Unlocked());
    m.def("layer_forward", &layer_forward, Unlocked());
    m.def("clear_scratch", &clear_scratch);
    m.def("set_get_plan", [](py::object f) { g_get_plan = new py::object(std::move(f)); });
}

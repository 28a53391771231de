// lib/torch_switchml_linear.so: the autograd node of ops/wgrad.py's FusedWgradLinear.
//
// Forward and backward of a small layer cost more on the host than on the GPU (256 x 512 x 512: 150 us
// against 20 us with the node in Python: its backward runs on the engine's thread, which has to get hold of
// the interpreter, and every step of it is a Python call). Here neither pass touches Python, unless the
// gradient is summed over several workers: that goes through the context's jobs, which `run` submits.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <memory>

#include "kernels/wgrad_gemm.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

void* CurrentStream() { return at::cuda::getCurrentCUDAStream().stream(); }

void Check(int rc, const char* what) {
  TORCH_CHECK(rc != -2, what, ": M and N must be multiples of 8 and all tensors 16-byte aligned");
  TORCH_CHECK(rc == 0, what, " failed (", rc, ")");
}

// What stays the same between the passes of a layer.
struct Plan : torch::CustomClassHolder {
  Tensor grad, error;  // fp32 [out, in], and the kernel's error flag
  std::unique_ptr<py::object> run;  // null with one worker; else called with (dy, x) in bf16
  ~Plan() override {
    if (!run) return;  // graphs are freed by threads that do not hold the interpreter's lock
    py::gil_scoped_acquire gil;
    run.reset();
  }
};

// `weight` and `bias` in the type that autocast computes in: fp32 to bf16 in one launch.
std::pair<Tensor, Tensor> CastWeights(const Tensor& weight, const Tensor& bias, at::ScalarType type) {
  const bool plain = type == at::kBFloat16 && weight.scalar_type() == at::kFloat && weight.is_contiguous() && weight.is_cuda() &&
                     weight.numel() > 0 && (!bias.defined() || (bias.scalar_type() == at::kFloat && bias.is_contiguous()));
  if (!plain) return {weight.to(type), bias.defined() ? bias.to(type) : Tensor()};
  Tensor w = at::empty_like(weight, weight.options().dtype(type));
  Tensor b = bias.defined() ? at::empty_like(bias, bias.options().dtype(type)) : Tensor();
  Check(switchml_cast_weights(weight.const_data_ptr<float>(), w.data_ptr(), weight.numel(),
                              b.defined() ? bias.const_data_ptr<float>() : nullptr, b.defined() ? b.data_ptr() : nullptr,
                              b.defined() ? bias.numel() : 0, CurrentStream()),
        "cast_weights");
  return {w, b};
}

class FusedLinear : public torch::autograd::Function<FusedLinear> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& weight_in, const std::optional<Tensor>& bias_in,
                        c10::intrusive_ptr<Plan> plan, std::optional<at::ScalarType> type) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
    const c10::cuda::OptionalCUDAGuard device(x_in.device());
    Tensor x = x_in, weight = weight_in, bias = bias_in.value_or(Tensor());
    ctx->saved_data["plan"] = c10::IValue::make_capsule(plan);
    ctx->saved_data["x_type"] = static_cast<int64_t>(x_in.scalar_type());
    ctx->saved_data["bias_type"] = bias.defined() ? static_cast<int64_t>(bias.scalar_type()) : int64_t(-1);
    if (type) {
      if (x.scalar_type() != *type) x = x.to(*type);
      std::tie(weight, bias) = CastWeights(weight, bias, *type);
      ctx->saved_data["weight"] = weight_in;  // only for gradients of gradients
    }
    ctx->save_for_backward({x, weight});
    return at::linear(x, weight, bias.defined() ? std::optional<Tensor>(bias) : std::nullopt);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor& dy = grads[0];
    const auto saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    Tensor weight = saved[1];
    const bool graph = at::GradMode::is_enabled();
    const c10::cuda::OptionalCUDAGuard device(x.device());
    if (graph && ctx->saved_data.count("weight")) weight = ctx->saved_data["weight"].toTensor().to(weight.scalar_type());
    const auto plan = c10::static_intrusive_pointer_cast<Plan>(ctx->saved_data["plan"].toCapsule());
    const Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    const Tensor dy2 = dy.dim() == 2 ? dy : dy.reshape({-1, dy.size(-1)});
    Tensor dx, dbias;
    if (ctx->needs_input_grad(0)) {
      dx = at::mm(dy2, weight.scalar_type() == dy2.scalar_type() ? weight : weight.to(dy2.scalar_type()));
      if (x.dim() != 2) dx = dx.reshape(x.sizes());
      const auto x_type = static_cast<at::ScalarType>(ctx->saved_data["x_type"].toInt());
      if (dx.scalar_type() != x_type) dx = dx.to(x_type);
    }
    {
      at::NoGradGuard no_grad;
      const Tensor dyl = dy2.to(at::kBFloat16).contiguous(), xl = x2.to(at::kBFloat16).contiguous();
      if (!plan->run) {
        // (The weight may be another one than the layer had when it was attached.)
        TORCH_CHECK(dyl.is_cuda() && xl.is_cuda() && dyl.size(1) * xl.size(1) == plan->grad.numel(), "the weight gradient is [",
                    dyl.size(1), ", ", xl.size(1), "], the buffer from attach() has ", plan->grad.numel(), " elements");
        Check(switchml_wgrad_gemm_auto(dyl.const_data_ptr(), xl.const_data_ptr(), plan->grad.data_ptr<float>(),
                                       static_cast<int>(dyl.size(1)), static_cast<int>(xl.size(1)), static_cast<int>(dyl.size(0)),
                                       plan->error.data_ptr<int>(), CurrentStream()),
              "wgrad_gemm");
      } else {
        py::gil_scoped_acquire gil;
        (*plan->run)(dyl, xl);
      }
    }
    const int64_t bias_type = ctx->saved_data["bias_type"].toInt();
    if (bias_type >= 0) {
      if (!graph && dy2.scalar_type() == at::kBFloat16 && dy2.is_contiguous() && dy2.size(1) % 8 == 0 &&
          (reinterpret_cast<uintptr_t>(dy2.const_data_ptr()) & 15) == 0) {
        dbias = at::empty({dy2.size(1)}, dy2.options().dtype(at::kFloat));
        Check(switchml_column_sums(dy2.const_data_ptr(), dbias.data_ptr<float>(), static_cast<int>(dy2.size(0)),
                                   static_cast<int>(dy2.size(1)), CurrentStream()),
              "column_sums");
      } else {
        dbias = dy2.sum(0);
      }
      if (dbias.scalar_type() != static_cast<at::ScalarType>(bias_type)) dbias = dbias.to(static_cast<at::ScalarType>(bias_type));
    }
    return {dx, Tensor(), dbias, Tensor(), Tensor()};
  }
};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Plan, c10::intrusive_ptr<Plan>>(m, "Plan").def(py::init([](Tensor grad, Tensor error, py::object run) {
    auto p = c10::make_intrusive<Plan>();
    p->grad = std::move(grad);
    p->error = std::move(error);
    if (!run.is_none()) p->run = std::make_unique<py::object>(std::move(run));
    return p;
  }));
  m.def("fused_linear", [](const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias, const c10::intrusive_ptr<Plan>& plan) {
    std::optional<at::ScalarType> type;
    if (at::autocast::is_autocast_enabled(at::kCUDA)) type = at::autocast::get_autocast_dtype(at::kCUDA);
    return FusedLinear::apply(x, weight, bias, plan, type);
  });
}

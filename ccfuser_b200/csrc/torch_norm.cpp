// LayerNorm as an autograd function in C++: what ops/norm.py did around the kernels of norm.cu, without the Python of an
// autograd.Function on either side. One forward and backward of 8192 x 2048 took 127 us of host time from Python for kernels that
// run 85 us when cold; one such pass among others took 129 us before and takes 85 now. The kernels and their launchers stay in
// libccfuser_b200.so, which this module is linked against.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <optional>

#include "norm.h"

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

std::atomic<long long> g_launches{0};

void check(int rc, const char* what) { TORCH_CHECK(rc == 0, what, " failed with code ", rc); }

// as the kernels read it: contiguous and on a 16-byte boundary (a view may begin anywhere)
at::Tensor packed(const at::Tensor& t) {
  const at::Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone();
}
at::Tensor rows_of(const at::Tensor& t, int64_t rows, int64_t d) { return packed(t.reshape({rows, d})); }

struct LayerNormFn : torch::autograd::Function<LayerNormFn> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& weight, const std::optional<at::Tensor>& bias,
                            const at::Tensor& status, double eps, int64_t wait_ns) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t d = x.size(-1), rows = x.numel() / d;
    const at::Tensor x2 = rows_of(x, rows, d), w = packed(weight);
    const at::Tensor b = bias.has_value() ? packed(*bias) : at::Tensor();
    const at::Tensor y = at::empty_like(x2);
    const auto f32 = x2.options().dtype(at::kFloat);
    const at::Tensor mean = at::empty({rows}, f32), rstd = at::empty({rows}, f32);
    check(ccf_layernorm_fwd(x2.data_ptr(), w.data_ptr(), b.defined() ? b.data_ptr() : nullptr, y.data_ptr(), mean.data_ptr<float>(),
                            rstd.data_ptr<float>(), static_cast<int>(rows), static_cast<int>(d), static_cast<float>(eps),
                            x.scalar_type() == at::kHalf, c10::cuda::getCurrentCUDAStream().stream()),
          "ccf_layernorm_fwd");
    ++g_launches;
    ctx->save_for_backward({x2, w, mean, rstd});
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["shape"] = x.sizes();
    ctx->saved_data["status"] = status;
    ctx->saved_data["wait_ns"] = wait_ns;
    return y.view(x.sizes());
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x2 = saved[0], &w = saved[1], &mean = saved[2], &rstd = saved[3];
    const c10::cuda::CUDAGuard guard(x2.device());
    const int64_t rows = x2.size(0), d = x2.size(1);
    const bool has_bias = ctx->saved_data["bias"].toBool();
    const at::Tensor dy = rows_of(grads[0], rows, d), dx = at::empty_like(x2), dg = at::empty_like(w);
    const at::Tensor db = has_bias ? at::empty_like(w) : at::Tensor();
    const int parts = ccf_layernorm_bwd_parts(static_cast<int>(rows), static_cast<int>(d));
    const at::Tensor part = at::empty({parts, 2, d}, x2.options().dtype(at::kFloat));
    check(ccf_layernorm_bwd(x2.data_ptr(), dy.data_ptr(), w.data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(), dx.data_ptr(),
                            part.data_ptr<float>(), dg.data_ptr(), has_bias ? db.data_ptr() : nullptr, static_cast<int>(rows),
                            static_cast<int>(d), x2.scalar_type() == at::kHalf, ctx->saved_data["status"].toTensor().data_ptr<int>(),
                            static_cast<unsigned long long>(ctx->saved_data["wait_ns"].toInt()),
                            c10::cuda::getCurrentCUDAStream().stream()),
          "ccf_layernorm_bwd");
    g_launches += 2;
    return {dx.view(ctx->saved_data["shape"].toIntVector()), dg, db, at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

}  // namespace

PYBIND11_MODULE(_ccf_torch, m) {
  m.def(
      "layer_norm",
      [](const at::Tensor& x, const at::Tensor& weight, const std::optional<at::Tensor>& bias, const at::Tensor& status, double eps,
         int64_t wait_ns) { return LayerNormFn::apply(x, weight, bias, status, eps, wait_ns); },
      py::call_guard<py::gil_scoped_release>());
  m.def("launches", [] { return g_launches.load(); });
}

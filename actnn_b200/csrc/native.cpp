// The host side of the hot entry points in C++: outputs are allocated, the Philox offset is drawn and the
// library is called without going through Python for each of them, and the mask-saving layers (ReLU,
// dropout, max pooling) are C++ autograd functions, so that their backward passes run without the interpreter.
//
// A training step of small layers is paced by the host: a bf16 / float16 layer makes about ten allocations and
// calls of 10 - 25 arguments in each direction.  Measured a pass, float16, forward + backward: batch norm of
// 128 x 256 x 14 x 14 217 -> 162 us (46 on the GPU), the bottleneck block at batch 256 2400 -> 2209, compress and
// decompress of 8 x 16 x 14 x 14 46 -> 37.
// The Python functions of actnn_b200.cpp_extension keep the checks and the argument forms; this file has no
// behaviour of its own.
#include <ATen/Functions.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CUDAGeneratorImpl.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <climits>
#include <mutex>

#include "../../include/actnn_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

int dtype_id(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return ACTNN_F32;
    case at::kHalf: return ACTNN_F16;
    case at::kBFloat16: return ACTNN_BF16;
    default: TORCH_CHECK(false, "actnn_b200: unsupported dtype ", c10::toString(t));
  }
}
void check(int status, const char* what) {
  TORCH_CHECK(status == ACTNN_OK, what, " failed: ", actnn_status_string(status), " (status " + std::to_string(status) + ")");
}
actnn_stream_t stream() { return (actnn_stream_t)at::cuda::getCurrentCUDAStream().stream(); }
void* ptr(const OptTensor& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// (seed, offset) from torch's default generator of the current device; advances the offset by one call.
std::pair<uint64_t, uint64_t> next_philox() {
  auto gen = at::cuda::detail::getDefaultCUDAGenerator();
  std::lock_guard<std::mutex> lock(gen.mutex());
  const uint64_t seed = gen.current_seed(), offset = gen.get_offset();
  gen.set_offset(offset + 4);
  return {seed, offset};
}
Tensor make(at::IntArrayRef shape, at::ScalarType t, const Tensor& like) {
  return at::empty(shape, like.options().dtype(t).memory_format(std::nullopt).requires_grad(false));
}
OptTensor as_f32(const OptTensor& t) {
  if (!t.has_value() || !t->defined()) return std::nullopt;
  return t->to(at::kFloat).contiguous();
}
at::ScalarType stat_type(const Tensor& data, bool bf16) { return bf16 ? at::kBFloat16 : data.scalar_type(); }

// ---------------------------------------------------------------------------------------- codec
// (packed, bits, scale, min, C, word_offsets); features < 0: data is [n, g, gs], whole groups
py::tuple compress_mixed(const Tensor& data, int64_t n, int64_t g, int64_t gs, int64_t features, double target_bits,
                         int64_t initial_bits, double range_factor, double coeff, const OptTensor& grad_scale,
                         bool stochastic, bool bf16_stats, const OptTensor& mn_in, const OptTensor& mx_in,
                         const OptTensor& ticket) {
  c10::cuda::CUDAGuard guard(data.device());
  const auto st = stat_type(data, bf16_stats);
  const int dt = dtype_id(data.scalar_type()), sd = dtype_id(st);
  const int64_t total = std::min(initial_bits * n, std::max((int64_t)target_bits, n));      // what the greedy ends with
  Tensor packed = make({(total * g * gs + 31) / 32}, at::kInt, data);
  Tensor scale = make({n, g, 1}, st, data), mn = make({n, g, 1}, st, data);
  Tensor bits = make({n}, at::kInt, data), offsets = make({n + 1}, at::kLong, data), C = make({n}, at::kFloat, data);
  uint64_t seed = 0, offset = 0;
  if (stochastic) std::tie(seed, offset) = next_philox();
  auto* words = packed.data_ptr<int32_t>();
  if (mn_in.has_value()) {
    check(actnn_compress_mixed_prestat_kept(data.data_ptr(), ptr(mn_in), ptr(mx_in), words, scale.data_ptr(), mn.data_ptr(),
                                            bits.data_ptr<int32_t>(), offsets.data_ptr<int64_t>(), C.data_ptr<float>(),
                                            ptr(ticket), n, g, gs, dt, sd, (float)range_factor, (float)coeff,
                                            (const float*)ptr(grad_scale), (int)initial_bits, target_bits, stochastic,
                                            nullptr, seed, offset, stream()),
          "actnn_compress_mixed_prestat_kept");
  } else {
    const int64_t bytes = actnn_compress_mixed_workspace(n, g, dt);
    Tensor ws = make({std::max<int64_t>(bytes, 256)}, at::kByte, data);
    if (features < 0)
      check(actnn_compress_mixed(data.data_ptr(), words, scale.data_ptr(), mn.data_ptr(), bits.data_ptr<int32_t>(),
                                 offsets.data_ptr<int64_t>(), C.data_ptr<float>(), ws.data_ptr(), bytes, n, g, gs, dt, sd,
                                 (float)range_factor, (float)coeff, (const float*)ptr(grad_scale), (int)initial_bits,
                                 target_bits, stochastic, nullptr, seed, offset, stream()),
            "actnn_compress_mixed");
    else
      check(actnn_compress_mixed_samples(data.data_ptr(), words, scale.data_ptr(), mn.data_ptr(),
                                         bits.data_ptr<int32_t>(), offsets.data_ptr<int64_t>(), C.data_ptr<float>(),
                                         ws.data_ptr(), bytes, n, features, dt, sd, (float)range_factor, (float)coeff,
                                         (const float*)ptr(grad_scale), (int)initial_bits, target_bits, stochastic,
                                         nullptr, seed, offset, stream()),
            "actnn_compress_mixed_samples");
  }
  return py::make_tuple(packed, bits, scale, mn, C, offsets);
}

Tensor unpack_mixed(const Tensor& packed, const Tensor& bits, const Tensor& offsets, const Tensor& scale, const Tensor& mn,
                    const std::vector<int64_t>& shape, int64_t n, int64_t g, int64_t gs, int64_t features,
                    const Tensor& like_dtype_of, bool as_float) {
  c10::cuda::CUDAGuard guard(packed.device());
  Tensor out = make(shape, as_float ? at::kFloat : like_dtype_of.scalar_type(), packed);
  const int dt = dtype_id(out.scalar_type()), sd = dtype_id(scale.scalar_type());
  if (features < 0)
    check(actnn_unpack_mixed(packed.data_ptr<int32_t>(), bits.data_ptr<int32_t>(), offsets.data_ptr<int64_t>(),
                             scale.data_ptr(), mn.data_ptr(), out.data_ptr(), n, g, gs, dt, sd, stream()),
          "actnn_unpack_mixed");
  else
    check(actnn_unpack_mixed_samples(packed.data_ptr<int32_t>(), bits.data_ptr<int32_t>(), offsets.data_ptr<int64_t>(),
                                     scale.data_ptr(), mn.data_ptr(), out.data_ptr(), n, features, dt, sd, stream()),
          "actnn_unpack_mixed_samples");
  return out;
}

// (packed, scale, min)
py::tuple compress_single(const Tensor& data, int64_t bits, bool stochastic, bool bf16_stats, int64_t bytes) {
  c10::cuda::CUDAGuard guard(data.device());
  const int64_t n = data.size(0), g = data.size(1), gs = data.size(2);
  const auto st = stat_type(data, bf16_stats);
  Tensor packed = make({bytes}, at::kChar, data), scale = make({n, g, 1}, st, data), mn = make({n, g, 1}, st, data);
  uint64_t seed = 0, offset = 0;
  if (stochastic) std::tie(seed, offset) = next_philox();
  check(actnn_compress_single(data.data_ptr(), (int)bits, packed.data_ptr<int8_t>(), scale.data_ptr(), mn.data_ptr(), nullptr,
                              n, g, gs, dtype_id(data.scalar_type()), dtype_id(st), stochastic, nullptr, seed, offset,
                              stream()),
        "actnn_compress_single");
  return py::make_tuple(packed, scale, mn);
}

// ---------------------------------------------------------------------------------------- batch norm
// (group minima, group maxima, mean, invstd), or None for a geometry that is not covered; `out`: room for the last two
py::object batch_norm_stats_minimax(const Tensor& x, const OptTensor& running_mean, const OptTensor& running_var,
                                    double momentum, double eps, const OptTensor& out) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t N = x.size(0), C = x.size(1), HW = N && C ? x.numel() / N / C : 0;
  const int64_t bytes = actnn_batch_norm_stats_minimax_workspace(N, C, HW);
  if (bytes < 0) return py::none();
  TORCH_CHECK(!out.has_value() || (out->scalar_type() == at::kFloat && out->is_contiguous() && out->numel() >= 2 * C &&
                                   out->device() == x.device()),
              "batch_norm_stats_minimax: out must be a contiguous float32 tensor of >= 2*C elements");
  const auto t = x.scalar_type();
  Tensor mn = make({N, C * HW / 256, 1}, t, x), mx = make({N, C * HW / 256, 1}, t, x);
  const Tensor both = out.has_value() ? out->view(-1) : make({2 * C}, at::kFloat, x);
  Tensor mean = both.narrow(0, 0, C), invstd = both.narrow(0, C, C);
  Tensor ws = make({bytes}, at::kByte, x);
  check(actnn_batch_norm_stats_minimax(x.data_ptr(), mn.data_ptr(), mx.data_ptr(), nullptr, nullptr,
                                       (float*)ptr(running_mean), (float*)ptr(running_var), mean.data_ptr<float>(),
                                       invstd.data_ptr<float>(), N, C, HW, momentum, eps, dtype_id(t), ws.data_ptr(),
                                       bytes, stream()),
        "actnn_batch_norm_stats_minimax");
  return py::make_tuple(mn, mx, mean, invstd);
}

// (y, packed, bits, scale, min, mean, invstd, word_offsets), or None for a geometry that is not covered
py::object batch_norm_forward(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
                              const OptTensor& running_var, double momentum, double eps, int64_t target_bits,
                              int64_t initial_bits, double range_factor, bool stochastic, const OptTensor& gmn,
                              const OptTensor& gmx, const OptTensor& mean_in, const OptTensor& invstd_in,
                              const Tensor& ticket) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t N = x.size(0), C = x.size(1), F = x.numel() / N, HW = F / C, G = (F + 255) / 256;
  const int dt = dtype_id(x.scalar_type());
  int64_t bytes = 0;
  if (actnn_batch_norm_codes_workspace(N, C, HW, dt, &bytes) != ACTNN_OK) return py::none();
  const auto st = stat_type(x, x.scalar_type() == at::kFloat);
  const int64_t total = std::min(initial_bits * N, std::max(target_bits, N));
  const OptTensor w = as_f32(weight), b = as_f32(bias);
  Tensor y = at::empty_like(x), packed = make({total * G * 8}, at::kInt, x);
  Tensor scale = make({N, G, 1}, st, x), mn = make({N, G, 1}, st, x), bits = make({N}, at::kInt, x);
  Tensor offsets = make({N + 1}, at::kLong, x), sens = make({N}, at::kFloat, x);
  Tensor mean = mean_in.has_value() ? *mean_in : make({C}, at::kFloat, x);
  Tensor invstd = invstd_in.has_value() ? *invstd_in : make({C}, at::kFloat, x);
  Tensor ws = make({bytes}, at::kByte, x);
  uint64_t seed = 0, offset = 0;
  if (stochastic) std::tie(seed, offset) = next_philox();
  check(actnn_batch_norm_codes_forward(
            x.data_ptr(), ptr(gmn), ptr(gmx), (const float*)ptr(w), (const float*)ptr(b), (float*)ptr(running_mean),
            (float*)ptr(running_var), y.data_ptr(), mean.data_ptr<float>(), invstd.data_ptr<float>(),
            packed.data_ptr<int32_t>(), scale.data_ptr(), mn.data_ptr(), bits.data_ptr<int32_t>(),
            offsets.data_ptr<int64_t>(), sens.data_ptr<float>(), N, C, HW, momentum, eps, dt, dtype_id(st),
            (float)range_factor, (int)initial_bits, (double)target_bits, stochastic, seed, offset, ticket.data_ptr(),
            ws.data_ptr(), bytes, stream()),
        "actnn_batch_norm_codes_forward");
  return py::make_tuple(y, packed, bits, scale, mn, mean, invstd, offsets);
}

// (grad_input, grad_weight, grad_bias), the last two in float32; None for a geometry that is not covered
py::object batch_norm_backward(const Tensor& packed, const Tensor& bits, const Tensor& offsets, const Tensor& scale,
                               const Tensor& mn, const std::vector<int64_t>& shape, const Tensor& grad_out, bool as_float,
                               const OptTensor& weight, const Tensor& mean, const Tensor& invstd) {
  c10::cuda::CUDAGuard guard(packed.device());
  int64_t F = 1;
  for (size_t i = 1; i < shape.size(); ++i) F *= shape[i];
  const int64_t N = shape[0], C = shape[1], HW = F / C;
  const auto t = as_float ? at::kFloat : scale.scalar_type();
  const int dt = dtype_id(t);
  int64_t bytes = 0;
  if (actnn_batch_norm_codes_workspace(N, C, HW, dt, &bytes) != ACTNN_OK) return py::none();
  const Tensor dy = grad_out.contiguous().to(t);
  const OptTensor w = as_f32(weight);
  Tensor dx = make(shape, t, packed), dw = make({C}, at::kFloat, packed), db = make({C}, at::kFloat, packed);
  Tensor ws = make({bytes}, at::kByte, packed);
  check(actnn_batch_norm_codes_backward(packed.data_ptr<int32_t>(), bits.data_ptr<int32_t>(), offsets.data_ptr<int64_t>(),
                                        scale.data_ptr(), mn.data_ptr(), dy.data_ptr(), (const float*)ptr(w),
                                        mean.data_ptr<float>(), invstd.data_ptr<float>(), dx.data_ptr(),
                                        dw.data_ptr<float>(), db.data_ptr<float>(), N, C, HW, dt,
                                        dtype_id(scale.scalar_type()), ws.data_ptr(), bytes, stream()),
        "actnn_batch_norm_codes_backward");
  return py::make_tuple(dx, dw, db);
}

// ---------------------------------------------------------------------------------------- small helpers
Tensor transpose16(const Tensor& x, bool to_channels_last) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t n = x.size(0), c = x.size(1), hw = x.size(2) * x.size(3);
  Tensor out = at::empty(x.sizes(), x.options().requires_grad(false).memory_format(
      to_channels_last ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous));
  check(actnn_transpose16(x.data_ptr(), out.data_ptr(), n, to_channels_last ? c : hw, to_channels_last ? hw : c, stream()),
        "actnn_transpose16");
  return out;
}

Tensor sample_sumsq(const Tensor& grad_in) {
  c10::cuda::CUDAGuard guard(grad_in.device());
  const Tensor grad = grad_in.contiguous();
  const int64_t n = grad.size(0);
  Tensor out = make({n}, at::kFloat, grad);
  check(actnn_sample_sumsq(grad.data_ptr(), out.data_ptr<float>(), n, grad.numel() / std::max<int64_t>(n, 1),
                           dtype_id(grad.scalar_type()), stream()),
        "actnn_sample_sumsq");
  return out;
}

// The mean of sample_sumsq over the samples (0-dimensional); at least one sample
Tensor mean_sample_sumsq(const Tensor& grad_in, const Tensor& ticket) {
  c10::cuda::CUDAGuard guard(grad_in.device());
  const Tensor grad = grad_in.contiguous();
  const int64_t n = grad.size(0);
  Tensor out = make({n}, at::kFloat, grad), mean = make({}, at::kFloat, grad);
  check(actnn_sample_sumsq_mean(grad.data_ptr(), out.data_ptr<float>(), mean.data_ptr<float>(), ticket.data_ptr(), n,
                                grad.numel() / n, dtype_id(grad.scalar_type()), stream()),
        "actnn_sample_sumsq_mean");
  return mean;
}

// A copy of a small device tensor on its way to the host: enqueued on the current stream when made, waited for (by the
// host, without the interpreter lock) in `wait`.
struct Readback {
  Tensor host;
  at::cuda::CUDAEvent copied;
  explicit Readback(const Tensor& t) {
    c10::cuda::CUDAGuard guard(t.device());
    host = t.to(at::TensorOptions().device(at::kCPU), /*non_blocking=*/true);        // pinned
    copied.record();
  }
  Tensor wait() {
    py::gil_scoped_release unlocked;
    copied.synchronize();
    return host;
  }
};

// ---------------------------------------------------------------------------------------- mask-saving layers
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

Tensor mask_like(const Tensor& x) { return make({(x.numel() + 31) / 32}, at::kInt, x); }

Tensor relu_backward(const Tensor& grad_in, const Tensor& mask) {
  c10::cuda::CUDAGuard guard(grad_in.device());
  const Tensor grad = grad_in.contiguous();
  Tensor out = at::empty_like(grad);
  check(actnn_relu_backward(grad.data_ptr(), mask.data_ptr<int32_t>(), out.data_ptr(), grad.numel(),
                            dtype_id(grad.scalar_type()), stream()),
        "actnn_relu_backward");
  return out;
}

// with_minmax: also min and max of every 256 outputs, not differentiable
struct Relu : torch::autograd::Function<Relu> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, bool with_minmax) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor y = at::empty_like(x), mask = mask_like(x);
    const int dt = dtype_id(x.scalar_type());
    variable_list out{y};
    if (with_minmax) {
      ctx->set_materialize_grads(false);               // no zero-filled gradients for the extrema; y's is filled below
      ctx->saved_data["sizes"] = x.sizes();
      ctx->saved_data["dtype"] = x.scalar_type();
      Tensor mn = make({x.numel() / 256}, x.scalar_type(), x), mx = make({x.numel() / 256}, x.scalar_type(), x);
      check(actnn_relu_forward_minimax(x.data_ptr(), y.data_ptr(), mask.data_ptr<int32_t>(), mn.data_ptr(), mx.data_ptr(),
                                       x.numel(), dt, stream()),
            "actnn_relu_forward_minimax");
      ctx->mark_non_differentiable({mn, mx});
      out.push_back(mn);
      out.push_back(mx);
    } else {
      check(actnn_relu_forward(x.data_ptr(), y.data_ptr(), mask.data_ptr<int32_t>(), x.numel(), dt, stream()),
            "actnn_relu_forward");
    }
    ctx->save_for_backward({mask});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor mask = ctx->get_saved_variables()[0];
    if (grads[0].defined()) return {relu_backward(grads[0], mask), Tensor()};
    // the layer above gave no gradient, which counts as zeros
    return {at::zeros(ctx->saved_data["sizes"].toIntVector(), mask.options().dtype(ctx->saved_data["dtype"].toScalarType())),
            Tensor()};
  }
};

struct Dropout : torch::autograd::Function<Dropout> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, double p) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor y = at::empty_like(x), mask = mask_like(x);
    const auto [seed, offset] = next_philox();
    check(actnn_dropout_forward(x.data_ptr(), y.data_ptr(), mask.data_ptr<int32_t>(), x.numel(), (float)p,
                                dtype_id(x.scalar_type()), nullptr, seed, offset, stream()),
          "actnn_dropout_forward");
    ctx->save_for_backward({mask});
    ctx->saved_data["p"] = p;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor grad = grads[0].contiguous(), mask = ctx->get_saved_variables()[0];
    c10::cuda::CUDAGuard guard(grad.device());
    Tensor out = at::empty_like(grad);
    check(actnn_dropout_backward(grad.data_ptr(), mask.data_ptr<int32_t>(), out.data_ptr(), grad.numel(),
                                 (float)ctx->saved_data["p"].toDouble(), dtype_id(grad.scalar_type()), stream()),
          "actnn_dropout_backward");
    return {out, Tensor()};
  }
};

struct MaxPool : torch::autograd::Function<MaxPool> {
  // geom: kernel, stride, padding, dilation, two values each
  static Tensor forward(AutogradContext* ctx, const Tensor& x, std::vector<int64_t> geom) {
    TORCH_CHECK(geom.size() == 8 && x.dim() == 4, "max_pool2d: a 4-dimensional input and eight geometry values are expected");
    int g[8];
    for (int i = 0; i < 8; ++i) {                      // the output size below divides by the stride
      const int64_t least = i == 4 || i == 5 ? 0 : 1;
      TORCH_CHECK(geom[i] >= least && geom[i] <= INT_MAX, "max_pool2d: kernel_size, stride and dilation must be positive and padding "
                  "not negative, got ", geom[i]);
      g[i] = (int)geom[i];
    }
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3);
    auto floordiv = [](int64_t a, int64_t b) { return a / b - (a % b != 0 && (a < 0) != (b < 0)); };
    const int64_t ho = floordiv(h + 2 * g[4] - (int64_t)g[6] * (g[0] - 1) - 1, g[2]) + 1;
    const int64_t wo = floordiv(w + 2 * g[5] - (int64_t)g[7] * (g[1] - 1) - 1, g[3]) + 1;
    Tensor y = make({n, c, ho, wo}, x.scalar_type(), x), idx = make({n, c, ho, wo}, at::kChar, x);
    check(actnn_max_pool2d_forward(x.data_ptr(), y.data_ptr(), idx.data_ptr<int8_t>(), n, c, h, w, g[0], g[1], g[2], g[3],
                                   g[4], g[5], g[6], g[7], dtype_id(x.scalar_type()), stream()),
          "actnn_max_pool2d_forward");
    ctx->save_for_backward({idx});
    ctx->saved_data["geom"] = geom;
    ctx->saved_data["shape"] = std::vector<int64_t>{n, c, h, w};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor grad = grads[0].contiguous(), idx = ctx->get_saved_variables()[0];
    c10::cuda::CUDAGuard guard(grad.device());
    const auto g = ctx->saved_data["geom"].toIntVector(), s = ctx->saved_data["shape"].toIntVector();
    Tensor out = make(s, grad.scalar_type(), grad);
    check(actnn_max_pool2d_backward(grad.data_ptr(), idx.data_ptr<int8_t>(), out.data_ptr(), s[0], s[1], s[2], s[3],
                                    (int)g[0], (int)g[1], (int)g[2], (int)g[3], (int)g[4], (int)g[5], (int)g[6], (int)g[7],
                                    dtype_id(grad.scalar_type()), stream()),
          "actnn_max_pool2d_backward");
    return {out, Tensor()};
  }
};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Readback>(m, "Readback").def(py::init<const Tensor&>()).def("wait", &Readback::wait);
  m.def("compress_mixed", &compress_mixed);
  m.def("unpack_mixed", &unpack_mixed);
  m.def("compress_single", &compress_single);
  m.def("batch_norm_stats_minimax", &batch_norm_stats_minimax);
  m.def("batch_norm_forward", &batch_norm_forward);
  m.def("batch_norm_backward", &batch_norm_backward);
  m.def("transpose16", &transpose16);
  m.def("sample_sumsq", &sample_sumsq);
  m.def("mean_sample_sumsq", &mean_sample_sumsq);
  m.def("relu", [](const Tensor& x) { return Relu::apply(x, false)[0]; });
  m.def("relu_minmax", [](const Tensor& x) { return Relu::apply(x, true); });
  m.def("dropout", [](const Tensor& x, double p) { return Dropout::apply(x, p); });
  m.def("max_pool2d", [](const Tensor& x, std::vector<int64_t> geom) { return MaxPool::apply(x, std::move(geom)); });
}

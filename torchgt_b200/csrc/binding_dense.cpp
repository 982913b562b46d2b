// Autograd nodes of the narrow linear layer (torchgt_b200/linear.py) and of LayerNorm (torchgt_b200/layer_norm.py):
// this library's kernels, issued without a trip through Python.
#include "binding.h"

#include <ATen/Context.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/stl.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/utils/pybind.h>

namespace tgt_host {
namespace {

using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

bool aligned(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

// contiguous, and copied when it is a view that starts off a 16-byte boundary (the kernels move 16 bytes at a time)
at::Tensor kernel_ready(const at::Tensor& t) {
  at::Tensor c = t.contiguous();
  return aligned(c) ? c : c.clone();
}

// a plain fp32 CUDA tensor, not a functorch wrapper, a dual number, a fake or a lazily negated view
bool plain(const at::Tensor& t, const at::Device& device) {
  return t.defined() && !at::isTensorSubclassLike(t) && t.is_cuda() && t.layout() == at::kStrided &&
         t.scalar_type() == at::kFloat && t.device() == device && !torch::autograd::isFwGradDefined(t) && !t.is_neg();
}

// The caller allowed TF32 products.
bool tf32_allowed() {
  return at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) ==
         at::Float32Precision::TF32;
}

// ---- which kernel takes a product ------------------------------------------------------------------------------------
// Device times in us, back to back in a graph: this library's kernels (linear_mma.cu, for few tiles linear_rows.cu) / PyTorch's
// operations.  Up to a thousand rows the library's rounding is kept: the calls are bound by the host.

// tiles of 128 rows x 64 columns of a result, what the tensor-core kernel's CTAs walk
int64_t tiles(int64_t rows, int64_t columns) { return (rows + 127) / 128 * ((columns + 63) / 64); }
// The longest reduction that is one launch of that kernel; longer ones need longer lists: 512 x 512 at 4,097 rows 47.9 / 51.9
// forward and 48.8 / 43.2 back, at 8,192 79 / 97 and 81 / 83, at 65,536 556 / 744 and 558 / 564; 1024 x 1024 at 1,100 rows 58
// / 50 and 61 / 44, at 8,192 282 / 358 and 280 / 321.
constexpr int64_t kOneLaunch = 384;
constexpr int64_t kManyTiles = 512;

// A single layer's x w^T + b, fp32.  The lines are those of an FMA kernel for every length; between them calls keep the
// library's rounding although the tensor cores are ahead of it now: 128 x 64 with a bias 18 / 14 at 16,384 rows then, 9.2 /
// 13.9 now; 64 x 64 without one 11.7 / 7.8 then, 6.5 / 6.9 now, 13 / 20.5 at 65,536; 64 x 4 with a bias 19 / 16 at 65,536
// then, 10 / 17 now; 256 x 256 with a bias 26.5 / 20.7 at 4,097 then, 14.9 / 19.2 now.  Inside: 64 x 64 with a bias, for which
// the library runs a second kernel, 3.6 / 5.5 at 1,100 rows, 4.2 / 6.4 at 4,097, 6.3 / 7.5 at 8,192, 13 / 32 at 65,536, 42 /
// 170 at 320,000; 128 x 64 5.5 / 6.6, 6.1 / 7.6, 18 / 41 and 70 / 215.  TF32: 3.6 / 3.2, 4.2 / 4.5, 6.3 / 3.5, 13 / 10.6, 42 /
// 34; 512 x 512 556 / 58 at 65,536.
bool layer_ahead(int64_t rows, int64_t in, int64_t out, bool bias) {
  if (tf32_allowed() || rows < 1024 || in > 128) return false;
  if (!bias) return in == 64 && out >= 32 && rows >= 65536;
  if (in == 128 && rows >= 8192 && rows < 32768) return false;
  return out >= 32 || rows < 32768;
}

// Up to 128 wide the blocks keep these kernels also where the library's take less device time, as long as a step is bound by
// launches, of which they need fewer.  fp32, any length: below 12,288 rows an input gradient of 64 x 64 is 6.2 / 4.4 us on the
// device, but a feed-forward block of 1,100 rows, forward and back, costs the host 104 us, with the library's input gradients
// 122.  TF32 allowed: short lists (128 x 128 at 8,192 rows 72 us on the device forward and back, 58 with the library's
// products, in 8 launches, not 11), and 64 x 64, where the device times are alike.
bool narrow_or_short(int64_t rows, int64_t in, int64_t out) {
  return in <= 128 && out <= 128 && (!tf32_allowed() || rows <= 8192 || in * out <= 64 * 64);
}

// A layer of the feed-forward block, with its activation or residual: 64 x 64 with gelu 4.8 / 7.5 at 1,100 rows, 9.1 / 13.4 at
// 16,384, 62 / 197 at 320,000; 128 x 64 with a residual 6.9 / 8.1, 11.9 / 16.2, 102 / 251; reductions over 128 from 80 tiles
// on (256 x 64 9.4 / 8.6 at 1,100 rows, 14.2 / 12.6 at 8,192, 14.7 / 18.1 at 10,240; 256 x 256 14.9 / 19.2 at 4,097).  TF32:
// 64 x 64 with gelu 4.8 / 5.2, 9.1 / 6.9, 18.4 / 16.3 at 65,536, 62 / 61; 64 x 128 28 / 22 and 115 / 91.
bool block_layer_ahead(int64_t rows, int64_t in, int64_t out) {
  if (rows < 1024) return false;
  if (tf32_allowed()) return narrow_or_short(rows, in, out);
  return in <= 128 || tiles(rows, out) >= (in > kOneLaunch ? kManyTiles : 80);
}

// Three products of one input.  fp32: 64 x 64 4.0 / 16.5, 100 / 510 at 320,000; 256 x 256 14.8 / 30 at 1,100, 1,490 / 3,430;
// 512 x 512 48 / 58 and 1,590 / 2,230 at 65,536.  TF32: 64 x 64 4.0 / 9.6, 8.3 / 10.5 at 8,192, 25 / 32 at 65,536, 100 / 103;
// 128 x 128 8.2 / 11.4, 14.5 / 18.3 at 8,192, 22.5 / 17.7 at 16,384; 64 x 128 9.9 / 13.2 at 8,192, 191 / 123 at 320,000;
// 192 x 192 22 / 16 at 4,097.
bool three_products_ahead(int64_t rows, int64_t in, int64_t out) {
  return !tf32_allowed() || narrow_or_short(rows, in, out);
}

// The sum of dy_i w_i, `out` being the reduction, for a single layer or in a block.  fp32, one: 64 x 64 6.2 / 4.4 at 8,192
// rows, 6.3 / 6.1 at 12,288, 6.4 / 7.1 at 16,384, 12.9 / 19.6 at 65,536, 41 / 87 at 320,000; 128 x 128 8.9 / 6.0 at 4,097, 9.0
// / 9.5 at 8,192; 256 outputs and 64 inputs 14.8 / 14.5 at 12,288, 37 / 48 at 65,536; 4 outputs 12.4 / 9.2 there.  With the
// derivative of relu or gelu 64 x 64 8.4 / 6.2 and 10.0 / 6.9 at 8,192, 8.9 / 9.4 and 10.5 / 10.5 at 16,384, 74 / 124 and 87 /
// 127 at 320,000.  Three: 64 x 64 11.8 / 11.6 at 1,100, 12.0 / 13.7 at 8,192, 106 / 305; 128 x 128 20.1 / 18.6 at 4,097, 20.3 /
// 30.5 at 8,192; 256 x 256 43.5 / 45.3 at 4,097, 1,860 / 2,520; 512 x 512 137 / 131 at 4,097, 233 / 258 at 8,192, 1,727 / 1,821
// at 65,536.  TF32: one 12.9 / 10.5 at 65,536; three of 64 x 64 12.0 / 10.7 at 8,192, 12.2 / 13.0 at 16,384, 106 / 164; 128
// inputs and 64 outputs 12.3 / 12.8 at 8,192, 197 / 199; 128 outputs 65 / 51 at 65,536; 256 inputs 87 / 65.
bool input_gradient_ahead(int64_t rows, int64_t out, int64_t in, size_t layers, bool block) {
  const int64_t have = tiles(rows, in);
  if (block && narrow_or_short(rows, in, out)) return true;
  if (tf32_allowed()) return layers > 1 && out <= 64 && in <= 128 && have >= 128;
  if (layers > 1) return out <= 64 || have >= (out > 256 ? kManyTiles : 128);
  return out >= 32 && (have >= (out > kOneLaunch ? kManyTiles : 128) || (rows >= 12288 && out <= kOneLaunch));
}

// dx = (sum of dy_i w_i) * act'(at gate), in the shape of `sizes`; gate: the activation's input, of relu its result.  All but w
// kernel_ready; below autograd.
at::Tensor input_gradient(const std::vector<at::Tensor>& dy, const std::vector<at::Tensor>& w, at::IntArrayRef sizes,
                          bool block, int act = TGT_ACT_NONE, const at::Tensor& gate = at::Tensor()) {
  const int64_t out = w[0].size(0), in = w[0].size(1), rows = dy[0].numel() / out;
  if (!input_gradient_ahead(rows, out, in, dy.size(), block)) {
    at::Tensor dx;
    for (size_t i = 0; i < dy.size(); ++i) {
      const at::Tensor d = dy[i].view({rows, out});
      if (i == 0) dx = at::mm(d, w[i]);
      else dx.addmm_(d, w[i]);
    }
    dx = dx.view(sizes);
    if (act == TGT_ACT_NONE) return dx;
    return act == TGT_ACT_RELU ? at::threshold_backward(dx, gate, 0) : at::gelu_backward(dx, gate);
  }
  std::vector<at::Tensor> kept;
  const float *from[3], *by[3];
  for (size_t i = 0; i < dy.size(); ++i) {
    kept.push_back(kernel_ready(w[i]));
    from[i] = fptr(dy[i]);
    by[i] = fptr(kept.back());
  }
  const at::Tensor dx = at::empty(sizes, dy[0].options());
  check(tgt_linear_input_grad_multi(from, by, int(dy.size()), rows, int(out), int(in), act, fptr(gate), fptr(dx),
                                    stream_of(dx)));
  return dx;
}

// dW = dY^T X and db = the sum of dY's rows where the gradient is itself differentiated (create_graph): the kernel's values,
// with what the two formulas' derivatives are as operations that can be recorded again.
struct ParameterGradientsBackward : public torch::autograd::Node {
  SavedVariable dy, x;

  variable_list apply(variable_list&& grads) override {
    const at::Tensor dy_ = dy.unpack(), x_ = x.unpack();
    variable_list result(2);
    if (grads[0].defined()) {
      if (task_should_compute_output(0)) result[0] = at::matmul(x_, grads[0].t());
      if (task_should_compute_output(1)) result[1] = at::matmul(dy_, grads[0]);
    }
    if (grads.size() > 1 && grads[1].defined() && task_should_compute_output(0)) {
      const at::Tensor rows = grads[1].expand_as(dy_);
      result[0] = result[0].defined() ? result[0] + rows : rows;
    }
    return result;
  }
  std::string name() const override { return "ParameterGradientsBackward"; }
  void release_variables() override {
    dy.reset_data();
    x.reset_data();
  }
};

// db may be undefined
void record_parameter_gradients(const at::Tensor& dw, const at::Tensor& db, const at::Tensor& dy, const at::Tensor& x) {
  if (!torch::autograd::compute_requires_grad(dy, x)) return;
  auto node = std::shared_ptr<ParameterGradientsBackward>(new ParameterGradientsBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(dy, x));
  node->dy = SavedVariable(dy, false);
  node->x = SavedVariable(x, false);
  torch::autograd::set_history(db.defined() ? variable_list{dw, db} : variable_list{dw}, node);
}

struct NarrowLinearBackward : public torch::autograd::Node {
  SavedVariable x, weight;
  bool has_bias = false;

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    if (!grads[0].defined()) return variable_list(3);
    const at::Tensor x_ = x.unpack(), w_ = weight.unpack();
    const c10::cuda::CUDAGuard guard(x_.device());
    at::Tensor dx, dw, db;
    const bool recorded = at::GradMode::is_enabled();     // a second-order gradient is wanted
    if (task_should_compute_output(0) && recorded) dx = at::matmul(grads[0], w_);
    kernels(grads[0], x_, w_, recorded, dx, dw, db);
    if (recorded && dw.defined()) record_parameter_gradients(dw, db, grads[0], x_);
    return {dx, dw, db};
  }
  void kernels(const at::Tensor& dy_, const at::Tensor& x_, const at::Tensor& w_, bool recorded, at::Tensor& dx, at::Tensor& dw,
               at::Tensor& db) {
    const at::AutoDispatchBelowADInplaceOrView below;
    const int64_t out = w_.size(0), in = w_.size(1);
    const at::Tensor dy = kernel_ready(dy_);
    const int64_t rows = dy.numel() / out;
    if (task_should_compute_output(0) && !recorded) dx = input_gradient({dy}, {w_}, x_.sizes(), false);
    if (task_should_compute_output(1) || (has_bias && task_should_compute_output(2))) {
      const at::Tensor xc = kernel_ready(x_);
      size_t bytes = 0;
      check(tgt_linear_wgrad_scratch_bytes(rows, int(in), int(out), &bytes));
      const at::Tensor scratch = at::empty({int64_t(bytes < 16 ? 16 : bytes)}, dy.options().dtype(at::kByte));
      dw = at::empty({out, in}, dy.options());
      if (has_bias) db = at::empty({out}, dy.options());
      check(tgt_linear_wgrad(fptr(dy), fptr(xc), rows, int(in), int(out), fptr(dw), has_bias ? fptr(db) : nullptr,
                             scratch.data_ptr(), scratch.numel(), stream_of(dy)));
    }
  }
  std::string name() const override { return "NarrowLinearBackward"; }
  void release_variables() override {
    x.reset_data();
    weight.reset_data();
  }
};

// The shapes of the kernels: whole 64-wide inputs, outputs in fours.  Everything else is the ATen operator.
bool eligible(const at::Tensor& x, const at::Tensor& w, const at::Tensor& bias) {
  if (!x.defined() || at::isTensorSubclassLike(x) || !plain(x, x.device()) || !plain(w, x.device())) return false;
  if (w.dim() != 2 || x.dim() < 1 || x.size(-1) != w.size(1) || x.numel() == 0) return false;
  const int64_t in = w.size(1), out = w.size(0);
  if (in % 64 != 0 || in < 64 || in > 1024 || out % 4 != 0 || out < 4 || out > 1024) return false;
  return !bias.defined() || (plain(bias, x.device()) && bias.dim() == 1 && bias.size(0) == out);
}

at::Tensor linear(const at::Tensor& x, const at::Tensor& w, const std::optional<at::Tensor>& bias_in) {
  const at::Tensor bias = bias_in.has_value() ? *bias_in : at::Tensor();
  if (!eligible(x, w, bias)) return at::linear(x, w, bias_in);
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / w.size(1);
  const bool library = !layer_ahead(rows, w.size(1), w.size(0), bias.defined());
  const bool record = torch::autograd::compute_requires_grad(x, w, bias);
  at::Tensor y;
  if (library && !record) return at::linear(x, w, bias_in);
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    if (library) {
      y = at::linear(x, w, bias_in);
    } else {
      auto sizes = x.sizes().vec();
      sizes.back() = w.size(0);
      y = at::empty(sizes, x.options());
      const at::Tensor xc = kernel_ready(x), wc = kernel_ready(w), bc = bias.defined() ? kernel_ready(bias) : bias;
      check(tgt_linear_rows(fptr(xc), fptr(wc), bc.defined() ? fptr(bc) : nullptr, rows, int(w.size(1)), int(w.size(0)),
                            fptr(y), stream_of(x)));
    }
  }
  if (record) {
    auto node = std::shared_ptr<NarrowLinearBackward>(new NarrowLinearBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, w, bias));
    node->has_bias = bias.defined();
    node->x = SavedVariable(x, false);
    node->weight = SavedVariable(w, false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---- three layers of one input: the query, key and value projections ---------------------------------------------
// Parameter gradients of up to three layers of one input, in one pass over it; db[i] may be null.
void parameter_gradients(const std::vector<at::Tensor>& dy, const at::Tensor& x, int64_t rows, int64_t in, int64_t out,
                         const std::vector<at::Tensor*>& dw, const std::vector<at::Tensor*>& db) {
  const int n = int(dy.size());
  // wider, the tiles of three gradients fill the chip once and a bit (512 x 512 at 8,192 rows 281 us together, 251 one by one)
  if (n > 1 && in * out > 384 * 384) {
    for (int i = 0; i < n; ++i) parameter_gradients({dy[i]}, x, rows, in, out, {dw[i]}, {db[i]});
    return;
  }
  size_t bytes = 0;
  check(tgt_linear_wgrad_multi_scratch_bytes(n, rows, int(in), int(out), &bytes));
  const at::Tensor scratch = at::empty({int64_t(bytes < 16 ? 16 : bytes)}, x.options().dtype(at::kByte));
  const float* from[3];
  float *w[3], *b[3];
  for (int i = 0; i < n; ++i) {
    from[i] = fptr(dy[i]);
    *dw[i] = at::empty({out, in}, x.options());
    w[i] = fptr(*dw[i]);
    if (db[i] != nullptr) *db[i] = at::empty({out}, x.options());
    b[i] = db[i] != nullptr ? fptr(*db[i]) : nullptr;
  }
  check(tgt_linear_wgrad_multi(from, fptr(x), n, rows, int(in), int(out), w, b, scratch.data_ptr(), scratch.numel(),
                               stream_of(x)));
}

struct NarrowLinear3Backward : public torch::autograd::Node {
  SavedVariable x, weight[3];
  bool has_bias = false;

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    const at::Tensor x_ = x.unpack();
    const bool recorded = at::GradMode::is_enabled();      // a second-order gradient is wanted
    variable_list result = kernels(grads, x_, recorded);
    for (int i = 0; recorded && i < 3; ++i)
      if (result[1 + 2 * i].defined()) record_parameter_gradients(result[1 + 2 * i], result[2 + 2 * i], grads[i], x_);
    return result;
  }
  variable_list kernels(const variable_list& grads, const at::Tensor& x_, bool recorded) {
    variable_list result(7);
    const c10::cuda::CUDAGuard guard(x_.device());
    const bool want_dx = task_should_compute_output(0);
    std::vector<at::Tensor> dy, w, dy_p;
    std::vector<at::Tensor*> dw, db;
    for (int i = 0; i < 3; ++i) {
      if (!grads[i].defined()) continue;
      const at::Tensor w_ = weight[i].unpack();
      if (want_dx && recorded) {
        const at::Tensor d = at::matmul(grads[i], w_);
        result[0] = result[0].defined() ? result[0] + d : d;
      }
      const at::AutoDispatchBelowADInplaceOrView below;
      dy.push_back(kernel_ready(grads[i]));
      w.push_back(w_);
      if (!task_should_compute_output(1 + 2 * i) && !(has_bias && task_should_compute_output(2 + 2 * i))) continue;
      dy_p.push_back(dy.back());
      dw.push_back(&result[1 + 2 * i]);
      db.push_back(has_bias ? &result[2 + 2 * i] : nullptr);
    }
    if (dy.empty()) return result;
    const at::AutoDispatchBelowADInplaceOrView below;
    const int64_t out = w[0].size(0), in = w[0].size(1), rows = x_.numel() / in;
    if (want_dx && !recorded) result[0] = input_gradient(dy, w, x_.sizes(), true);
    if (!dy_p.empty()) parameter_gradients(dy_p, kernel_ready(x_), rows, in, out, dw, db);
    return result;
  }
  std::string name() const override { return "NarrowLinear3Backward"; }
  void release_variables() override {
    x.reset_data();
    for (SavedVariable& w : weight) w.reset_data();
  }
};

// {x w_i^T + b_i}
std::vector<at::Tensor> linear3(const at::Tensor& x, const std::vector<at::Tensor>& w,
                                const std::vector<std::optional<at::Tensor>>& bias_in) {
  TORCH_CHECK(w.size() == 3 && bias_in.size() == 3, "linear3 takes three layers");
  std::vector<at::Tensor> bias;
  bool together = true;
  for (int i = 0; i < 3; ++i) {
    bias.push_back(bias_in[i].has_value() ? *bias_in[i] : at::Tensor());
    together = together && eligible(x, w[i], bias[i]) && w[i].sizes() == w[0].sizes() && bias[i].defined() == bias[0].defined();
  }
  if (!together || x.numel() / w[0].size(1) < 1024)
    return {tgt_host::linear(x, w[0], bias_in[0]), tgt_host::linear(x, w[1], bias_in[1]), tgt_host::linear(x, w[2], bias_in[2])};
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t out = w[0].size(0), in = w[0].size(1), rows = x.numel() / in;
  variable_list y;
  if (!three_products_ahead(rows, in, out)) {
    const at::AutoDispatchBelowADInplaceOrView below;
    for (int i = 0; i < 3; ++i) y.push_back(at::linear(x, w[i], bias_in[i]));
  } else {
    const at::AutoDispatchBelowADInplaceOrView below;
    const at::Tensor xc = kernel_ready(x);
    auto sizes = x.sizes().vec();
    sizes.back() = out;
    std::vector<at::Tensor> kept;      // copies, while the launch needs them
    const float *by[3], *b[3];
    float* c[3];
    for (int i = 0; i < 3; ++i) {
      kept.push_back(kernel_ready(w[i]));
      by[i] = fptr(kept.back());
      if (bias[i].defined()) kept.push_back(kernel_ready(bias[i]));
      b[i] = bias[i].defined() ? fptr(kept.back()) : nullptr;
      y.push_back(at::empty(sizes, x.options()));
      c[i] = fptr(y[i]);
    }
    check(tgt_linear_rows_multi(fptr(xc), by, b, 3, rows, int(in), int(out), TGT_ACT_NONE, nullptr, nullptr, c, stream_of(x)));
  }
  if (torch::autograd::compute_requires_grad(x, w[0], w[1], w[2], bias[0], bias[1], bias[2])) {
    auto node = std::shared_ptr<NarrowLinear3Backward>(new NarrowLinear3Backward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, w[0], bias[0], w[1], bias[1], w[2], bias[2]));
    node->has_bias = bias[0].defined();
    node->x = SavedVariable(x, false);
    for (int i = 0; i < 3; ++i) node->weight[i] = SavedVariable(w[i], false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---- feed-forward block: act(x w1^T + b1) w2^T + b2 (+ residual) ---------------------------------------------------
struct FeedForwardBackward : public torch::autograd::Node {
  SavedVariable x, w1, b1, w2, hidden, gate;   // gate: the activation's input (relu: its result says enough)
  int act = TGT_ACT_NONE;
  bool with_residual = false;

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  // With create_graph the gradient is itself differentiated: the block's formula as recorded operations.
  variable_list recorded(const at::Tensor& dy, const at::Tensor& x_, const at::Tensor& w1_, const at::Tensor& w2_) {
    const at::Tensor z = at::linear(x_, w1_, b1.unpack());
    const at::Tensor h = act == TGT_ACT_RELU ? at::relu(z) : at::gelu(z);
    const at::Tensor dh = at::matmul(dy, w2_);
    const at::Tensor dz = act == TGT_ACT_RELU ? dh * (z > 0).to(dh.scalar_type()) : at::gelu_backward(dh, z);
    auto flat = [](const at::Tensor& t) { return t.reshape({-1, t.size(-1)}); };
    return {at::matmul(dz, w1_), at::matmul(flat(dz).t(), flat(x_)), flat(dz).sum(0), at::matmul(flat(dy).t(), flat(h)),
            flat(dy).sum(0), with_residual ? dy : at::Tensor()};
  }
  variable_list backward(const variable_list& grads) {
    variable_list result(6);
    if (!grads[0].defined()) return result;
    const at::Tensor x_ = x.unpack(), w1_ = w1.unpack(), w2_ = w2.unpack();
    if (at::GradMode::is_enabled()) return recorded(grads[0], x_, w1_, w2_);
    if (with_residual) result[5] = grads[0];
    const at::Tensor h = hidden.unpack(), gate_ = act == TGT_ACT_RELU ? h : gate.unpack();
    const c10::cuda::CUDAGuard guard(x_.device());
    const at::AutoDispatchBelowADInplaceOrView below;
    const at::Tensor dy = kernel_ready(grads[0]), hc = kernel_ready(h), gc = kernel_ready(gate_);
    const int64_t in = w1_.size(1), mid = w1_.size(0), out = w2_.size(0), rows = x_.numel() / in;
    if (task_should_compute_output(3) || task_should_compute_output(4))
      parameter_gradients({dy}, hc, rows, mid, out, {&result[3]}, {&result[4]});
    const bool first = task_should_compute_output(1) || task_should_compute_output(2);
    if (!first && !task_should_compute_output(0)) return result;
    const at::Tensor dz = input_gradient({dy}, {w2_}, h.sizes(), true, act, gc);
    if (first) parameter_gradients({dz}, kernel_ready(x_), rows, in, mid, {&result[1]}, {&result[2]});
    if (task_should_compute_output(0)) result[0] = input_gradient({dz}, {w1_}, x_.sizes(), true);
    return result;
  }
  std::string name() const override { return "FeedForwardBackward"; }
  void release_variables() override {
    for (SavedVariable* v : {&x, &w1, &b1, &w2, &hidden, &gate}) v->reset_data();
  }
};

bool feed_forward_eligible(const at::Tensor& x, const at::Tensor& w1, const at::Tensor& b1, const at::Tensor& w2,
                           const at::Tensor& b2, const at::Tensor& residual) {
  if (!b1.defined() || !b2.defined() || !eligible(x, w1, b1) || !plain(w2, x.device()) || !plain(b2, x.device()))
    return false;
  if (w2.dim() != 2 || w2.size(1) != w1.size(0) || b2.dim() != 1 || b2.size(0) != w2.size(0)) return false;
  const int64_t mid = w2.size(1), out = w2.size(0);
  const int64_t rows = x.numel() / w1.size(1);
  if (mid % 64 != 0 || mid > 1024 || out % 4 != 0 || out < 4 || out > 1024) return false;
  // one by one otherwise: a node of the library's products would save nothing
  if (!block_layer_ahead(rows, w1.size(1), mid) || !block_layer_ahead(rows, mid, out)) return false;
  return !residual.defined() || (plain(residual, x.device()) && out == w1.size(1) && residual.sizes() == x.sizes());
}

at::Tensor feed_forward(const at::Tensor& x, const at::Tensor& w1, const at::Tensor& b1, const at::Tensor& w2,
                        const at::Tensor& b2, const std::string& activation, const std::optional<at::Tensor>& residual_in) {
  const at::Tensor residual = residual_in.has_value() ? *residual_in : at::Tensor();
  TORCH_CHECK(activation == "relu" || activation == "gelu", "feed_forward knows relu and gelu, not ", activation);
  const int act = activation == "relu" ? TGT_ACT_RELU : TGT_ACT_GELU;
  if (!feed_forward_eligible(x, w1, b1, w2, b2, residual)) {
    const at::Tensor z = tgt_host::linear(x, w1, b1);
    const at::Tensor y = tgt_host::linear(act == TGT_ACT_RELU ? at::relu(z) : at::gelu(z), w2, b2);
    return residual.defined() ? residual + y : y;
  }
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t in = w1.size(1), mid = w1.size(0), out = w2.size(0), rows = x.numel() / in;
  const bool record = torch::autograd::compute_requires_grad(x, w1, b1, w2, b2, residual);
  at::Tensor y, h, z;
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    const at::Tensor xc = kernel_ready(x), w1c = kernel_ready(w1), b1c = kernel_ready(b1), w2c = kernel_ready(w2),
                     b2c = kernel_ready(b2), rc = residual.defined() ? kernel_ready(residual) : residual;
    auto sizes = x.sizes().vec();
    sizes.back() = mid;
    h = at::empty(sizes, x.options());
    if (record && act == TGT_ACT_GELU) z = at::empty(sizes, x.options());
    sizes.back() = out;
    y = at::empty(sizes, x.options());
    const float *by = fptr(w1c), *b = fptr(b1c);
    float* c = fptr(h);
    check(tgt_linear_rows_multi(fptr(xc), &by, &b, 1, rows, int(in), int(mid), act, fptr(z), nullptr, &c, stream_of(x)));
    by = fptr(w2c); b = fptr(b2c); c = fptr(y);
    check(tgt_linear_rows_multi(fptr(h), &by, &b, 1, rows, int(mid), int(out), TGT_ACT_NONE, nullptr,
                                rc.defined() ? fptr(rc) : nullptr, &c, stream_of(x)));
  }
  if (record) {
    auto node = std::shared_ptr<FeedForwardBackward>(new FeedForwardBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, w1, b1, w2, b2, residual));
    node->act = act;
    node->with_residual = residual.defined();
    node->x = SavedVariable(x, false);
    node->w1 = SavedVariable(w1, false);
    node->b1 = SavedVariable(b1, false);
    node->w2 = SavedVariable(w2, false);
    node->hidden = SavedVariable(h, false);
    node->gate = SavedVariable(z, false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---- sum of embedding vectors ---------------------------------------------------------------------------------------
struct EmbeddingSumBackward : public torch::autograd::Node {
  SavedVariable ids;
  int64_t n_table = 0, hidden = 0, padding = -1;

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    if (!grads[0].defined()) return variable_list(1);
    const at::Tensor ids_ = ids.unpack();
    // a second-order gradient is wanted, or many gradients at once (is_grads_batched): the library's recorded operation
    if (at::GradMode::is_enabled() || at::isTensorSubclassLike(grads[0])) {
      auto sizes = ids_.sizes().vec();
      sizes.push_back(hidden);
      return {at::embedding_dense_backward(grads[0].unsqueeze(-2).expand(sizes), ids_, n_table, padding, false)};
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(ids_.device());
    const at::Tensor dy = kernel_ready(grads[0]), ic = ids_.contiguous();
    const int64_t features = ids_.size(-1), rows = ids_.numel() / features;
    size_t bytes = 0;
    check(tgt_embedding_sum_grad_scratch_bytes(n_table, int(hidden), rows, int(features), &bytes));
    const at::Tensor scratch = at::empty({int64_t(bytes)}, dy.options().dtype(at::kByte));
    const at::Tensor dtable = at::empty({n_table, hidden}, dy.options());
    check(tgt_embedding_sum_grad(fptr(dy), static_cast<const int64_t*>(ptr(ic)), rows, int(features), n_table, int(hidden),
                                 padding, fptr(dtable), scratch.data_ptr(), scratch.numel(), stream_of(dy)));
    return {dtable};
  }
  std::string name() const override { return "EmbeddingSumBackward"; }
  void release_variables() override { ids.reset_data(); }
};

// embedding(ids).sum(-2)
at::Tensor embedding_sum(const at::Tensor& table, const at::Tensor& ids, int64_t padding) {
  constexpr int64_t kMost = int64_t(1) << 26;
  const bool own = ids.defined() && table.defined() && !at::isTensorSubclassLike(ids) && plain(table, ids.device()) &&
                   ids.is_cuda() && ids.layout() == at::kStrided && ids.scalar_type() == at::kLong && ids.dim() >= 1 &&
                   ids.numel() > 0 && table.dim() == 2 &&
                   (table.size(1) == 32 || table.size(1) == 64 || table.size(1) == 128) && table.size(0) >= 1 &&
                   table.size(0) < kMost && ids.size(-1) <= 1024 && ids.numel() / ids.size(-1) < kMost &&
                   ids.numel() < (int64_t(1) << 31) - 1;
  if (!own) return at::embedding(table, ids, padding).sum(-2);
  const c10::cuda::CUDAGuard guard(table.device());
  const int64_t features = ids.size(-1), rows = ids.numel() / features, hidden = table.size(1);
  at::Tensor out;
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    const at::Tensor tc = kernel_ready(table), ic = ids.contiguous();
    auto sizes = ids.sizes().vec();
    sizes.back() = hidden;
    out = at::empty(sizes, table.options());
    check(tgt_embedding_sum(fptr(tc), table.size(0), int(hidden), static_cast<const int64_t*>(ptr(ic)), rows, int(features),
                            fptr(out), stream_of(table)));
  }
  if (torch::autograd::compute_requires_grad(table)) {
    auto node = std::shared_ptr<EmbeddingSumBackward>(new EmbeddingSumBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(table));
    node->ids = SavedVariable(ids, false);
    node->n_table = table.size(0);
    node->hidden = hidden;
    node->padding = padding;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ---- LayerNorm, with the residual addition in front of it ------------------------------------------------------
// Outputs: the normalised rows and, with a residual, x + residual.
struct LayerNormRowsBackward : public torch::autograd::Node {
  SavedVariable normalised, weight, stats;   // the norm's input: x, or the output x + residual
  bool with_residual = false;
  double eps = 0;

  // With create_graph the gradient is itself differentiated: the formula as recorded operations.
  variable_list recorded(const at::Tensor& dy, const at::Tensor& ds, const at::Tensor& x, const at::Tensor& w) {
    const int64_t hidden = w.numel();
    const at::Tensor d = x - x.mean(-1, true), rstd = (d * d).mean(-1, true).add(eps).rsqrt(), xhat = d * rstd;
    const at::Tensor g = dy * w;
    at::Tensor dx = rstd * (g - g.mean(-1, true) - xhat * (g * xhat).mean(-1, true));
    if (ds.defined()) dx = dx + ds;
    return {dx, with_residual ? dx : at::Tensor(), (dy * xhat).reshape({-1, hidden}).sum(0),
            dy.reshape({-1, hidden}).sum(0)};
  }

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    const at::Tensor ds = with_residual ? grads[1] : at::Tensor();
    if (!grads[0].defined()) return {ds, ds, at::Tensor(), at::Tensor()};   // only x + residual was used
    const at::Tensor x = with_residual ? normalised.unpack(shared_from_this()) : normalised.unpack();
    const at::Tensor w = weight.unpack(), stats_ = stats.unpack();
    if (at::GradMode::is_enabled()) return recorded(grads[0], ds, x, w);
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(x.device());
    const at::Tensor dy = kernel_ready(grads[0]), xc = kernel_ready(x), wc = kernel_ready(w);
    const at::Tensor dsum = ds.defined() ? kernel_ready(ds) : ds;
    const int64_t hidden = w.numel(), rows = x.numel() / hidden;
    const at::Tensor dx = at::empty(x.sizes(), dy.options());
    const at::Tensor dgamma = at::empty(w.sizes(), dy.options()), dbeta = at::empty(w.sizes(), dy.options());
    size_t bytes = 0;
    check(tgt_layer_norm_bwd_scratch_bytes(rows, int(hidden), &bytes));
    const at::Tensor scratch = at::empty({int64_t(bytes < 16 ? 16 : bytes)}, dy.options().dtype(at::kByte));
    check(tgt_add_layer_norm_bwd(fptr(dy), dsum.defined() ? fptr(dsum) : nullptr, fptr(xc), fptr(wc), fptr(stats_), rows,
                                 int(hidden), fptr(dx), fptr(dgamma), fptr(dbeta), scratch.data_ptr(), scratch.numel(),
                                 stream_of(dy)));
    return {dx, with_residual ? dx : at::Tensor(), dgamma, dbeta};
  }
  std::string name() const override { return "LayerNormRowsBackward"; }
  void release_variables() override {
    normalised.reset_data();
    weight.reset_data();
    stats.reset_data();
  }
};

bool norm_eligible(const at::Tensor& x, const at::Tensor& residual, const at::Tensor& w, const at::Tensor& b) {
  if (!x.defined() || at::isTensorSubclassLike(x)) return false;
  const at::Device device = x.device();
  if (!plain(x, device) || !plain(w, device) || !plain(b, device)) return false;
  const int64_t hidden = w.numel();
  if (w.dim() != 1 || b.dim() != 1 || b.numel() != hidden || x.dim() < 1 || x.size(-1) != hidden || x.numel() == 0 ||
      hidden % 4 != 0 || hidden < 4 || hidden > 512)
    return false;
  return !residual.defined() || (plain(residual, device) && residual.sizes() == x.sizes());
}

// {norm of x (+ residual), x + residual or nothing}; the sum is left out when nobody wants it
std::pair<at::Tensor, std::optional<at::Tensor>> add_layer_norm(const at::Tensor& x,
                                                                const std::optional<at::Tensor>& residual_in,
                                                                const at::Tensor& w, const at::Tensor& b, double eps,
                                                                bool want_sum) {
  const at::Tensor residual = residual_in.has_value() ? *residual_in : at::Tensor();
  if (!norm_eligible(x, residual, w, b)) {
    const at::Tensor s = residual.defined() ? x + residual : x;
    return {at::layer_norm(s, w.sizes(), w, b, eps), residual.defined() ? std::optional<at::Tensor>(s) : std::nullopt};
  }
  const c10::cuda::CUDAGuard guard(x.device());
  const bool record = torch::autograd::compute_requires_grad(x, residual, w, b);
  const int64_t hidden = w.numel(), rows = x.numel() / hidden;
  at::Tensor y, sum, stats;
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    const at::Tensor xc = kernel_ready(x), wc = kernel_ready(w), bc = kernel_ready(b);
    const at::Tensor rc = residual.defined() ? kernel_ready(residual) : residual;
    y = at::empty(x.sizes(), x.options());
    if (residual.defined() && (want_sum || record)) sum = at::empty(x.sizes(), x.options());
    if (record) stats = at::empty({rows, 2}, x.options());
    check(tgt_add_layer_norm_fwd(fptr(xc), rc.defined() ? fptr(rc) : nullptr, fptr(wc), fptr(bc), float(eps), rows,
                                 int(hidden), sum.defined() ? fptr(sum) : nullptr, fptr(y), record ? fptr(stats) : nullptr,
                                 stream_of(x)));
  }
  if (record) {
    auto node = std::shared_ptr<LayerNormRowsBackward>(new LayerNormRowsBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, residual, w, b));
    node->with_residual = residual.defined();
    node->eps = eps;
    node->stats = SavedVariable(stats, false);
    node->weight = SavedVariable(w, false);
    if (residual.defined()) {
      torch::autograd::set_history(variable_list{y, sum}, node);
      node->normalised = SavedVariable(sum, true);
    } else {
      torch::autograd::set_history(y, node);
      node->normalised = SavedVariable(x, false);
    }
  }
  return {y, sum.defined() ? std::optional<at::Tensor>(sum) : std::nullopt};
}

at::Tensor layer_norm(const at::Tensor& x, const at::Tensor& w, const at::Tensor& b, double eps) {
  return add_layer_norm(x, std::nullopt, w, b, eps, false).first;
}

// ---- a pre-norm encoder layer ----------------------------------------------------------------------------------------
// What torchgt_b200/graphormer.py's EncoderLayer does with its modules on one rank, the same operations in the same order,
// without going back to Python between them: a layer's nine launches on 4,096 rows cost 100 us of host time one by one from
// the modules.  The attention takes the projections as they are, so no views stand between the nodes.  `p`: weight and bias (or
// none) of the first norm, the query, key, value and output projections, the second norm and the two feed-forward layers.
// Nothing, and nothing launched, where the projections are not heads * head_dim wide: the modules say what is wrong.
std::optional<at::Tensor> encoder_layer(const at::Tensor& x, const std::shared_ptr<Graph>& graph, int heads, int head_dim,
                         const std::vector<std::optional<at::Tensor>>& p, double eps, double ffn_eps) {
  TORCH_CHECK(p.size() == 16, "encoder_layer takes eight weights and their biases");
  TORCH_CHECK(x.numel() == graph->n_rows * x.size(-1), "x and the graph have different numbers of rows");
  auto weight = [&p](int i) -> const at::Tensor& { return *p[2 * i]; };
  for (int i = 1; i <= 3; ++i)
    if (weight(i).dim() != 2 || weight(i).size(0) != int64_t(heads) * head_dim) return std::nullopt;
  const at::Tensor y = layer_norm(x, weight(0), *p[1], eps);
  const std::vector<at::Tensor> qkv = linear3(y, {weight(1), weight(2), weight(3)}, {p[3], p[5], p[7]});
  const at::Tensor attended = attention_over_rows(qkv[0], qkv[1], qkv[2], at::Tensor(), graph, heads, head_dim);
  const auto [normed, sum] = add_layer_norm(x, tgt_host::linear(attended, weight(4), p[9]), weight(5), *p[11], ffn_eps, true);
  return feed_forward(normed, weight(6), *p[13], weight(7), *p[15], "gelu", sum);
}

}  // namespace

void bind_dense(pybind11::module_& m) {
  m.def("linear", &linear, Unlocked());
  m.def("linear3", &linear3, Unlocked());
  m.def("embedding_sum", &embedding_sum, Unlocked());
  m.def("feed_forward", &feed_forward, Unlocked());
  m.def("layer_norm", &layer_norm, Unlocked());
  m.def("add_layer_norm", &add_layer_norm, Unlocked());
  m.def("encoder_layer", &encoder_layer, Unlocked());
}

}  // namespace tgt_host

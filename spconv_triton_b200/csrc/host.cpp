// Host side of the layers: rulebook, allocations, kernels and the autograd node of a sparse convolution or
// pooling layer in one call each, over the C ABI of this library.
//
// Written in Python, these steps were 40 - 100 us of interpreter, ctypes and allocator calls a layer and
// direction, more than the kernels of a layer of a few thousand voxels take.  Here a layer is two calls (its
// rulebook, its arithmetic) that release the interpreter lock; backward never enters Python.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <pybind11/stl.h>

#include <memory>
#include <mutex>

#include "../../include/spconv_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Failure : std::runtime_error {
  int status;
  Failure(int s, const std::string& m) : std::runtime_error(m), status(s) {}
};
void check(int status) {
  if (status != SPC_OK) throw Failure(status, spc_last_error());
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// An operand as the kernels read it, in 16-byte words: contiguous (a view that starts elsewhere is copied; the
// CUDA-core kernels that take such views read column-major tables, which are not made for the others).
Tensor operand(const Tensor& t) {
  const Tensor c = t.contiguous();
  return (reinterpret_cast<uintptr_t>(c.const_data_ptr()) & 15u) != 0 ? c.clone() : c;
}
// Refuses operands of several GPUs: a kernel would be handed another GPU's addresses.
void on_one_device(std::initializer_list<const Tensor*> ts) {
  const Tensor& first = **ts.begin();
  for (const Tensor* t : ts)
    if (t->defined() && t->device() != first.device())
      throw pybind11::value_error("expected all tensors on " + first.device().str() + ", found one on " + t->device().str());
}
int32_t* ints(const Tensor& t) { return t.defined() ? t.data_ptr<int32_t>() : nullptr; }
void* data(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
int code_of(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return SPC_F16;
    case at::kBFloat16: return SPC_BF16;
    case at::kFloat: return SPC_F32;
    case at::kDouble: return SPC_F64;
    default: throw Failure(SPC_ERR_UNSUPPORTED, std::string("dtype ") + c10::toString(t) + " is not supported by spconv_triton_b200");
  }
}

// ---- rulebooks -------------------------------------------------------------------------------------------

struct Geometry {
  spc_geometry g{};
  int kv = 1, kvp = 4;
  bool subm = false;
  std::vector<int64_t> out_shape;
};

std::shared_ptr<Geometry> make_geometry(int batch, const std::vector<int>& in, const std::vector<int>& out,
                                        const std::vector<int>& ksize, const std::vector<int>& stride,
                                        const std::vector<int>& pad, const std::vector<int>& dil, bool subm, bool transpose) {
  auto q = std::make_shared<Geometry>();
  q->g.ndim = static_cast<int32_t>(in.size());
  if (in.empty() || in.size() > SPC_MAX_NDIM) throw Failure(SPC_ERR_INVALID_ARGUMENT, "geometry: bad number of dimensions");
  q->g.batch_size = batch;
  q->g.subm = subm;
  q->g.transpose = transpose;
  for (size_t d = 0; d < in.size(); ++d) {
    q->g.in_shape[d] = in[d];
    q->g.out_shape[d] = out.at(d);
    q->g.ksize[d] = ksize.at(d);
    q->g.stride[d] = stride.at(d);
    q->g.padding[d] = pad.at(d);
    q->g.dilation[d] = dil.at(d);
    q->kv *= ksize[d];
    q->out_shape.push_back(out[d]);
  }
  q->kvp = (q->kv + 3) & ~3;
  q->subm = subm;
  return q;
}

// Rows from which on the GEMM's row order is worth its sort: with a tile or less there is nothing to group.
constexpr int64_t kOrderRows = 256;
// ... and up to which the order that a submanifold rulebook was built without is made when a layer wants it.
constexpr int64_t kLateOrderRows = 8192;

// The tables of one rulebook, output side and input side, made as they are asked for.  The kernels read the
// row-major tables; the column-major ones serve the CUDA-core and weight-gradient kernels.
//
// Whoever builds a rulebook orders its streams as for any tensor.  Tables made later are made on the stream of the
// call that asks first; `late` lets a call on another stream wait for them.
struct Rulebook {
  std::shared_ptr<Geometry> geo;
  Tensor indices, out_indices, workspace;
  int64_t n_in = 0, n_out = 0;
  struct Side {
    Tensor rm, cm, order;
  };
  struct Late {
    c10::optional<c10::cuda::CUDAStream> stream;
    at::cuda::CUDAEvent made;
  };
  Side fwd, bwd;
  Late late_fwd, late_bwd;
  bool captured = false;  // by a graph, whose replays read the tables and what it makes tables from
  mutable std::mutex lock;

  bool subm() const { return geo->subm; }
  Tensor make(int64_t a, int64_t b) const { return at::empty({a, b}, indices.options()); }
  bool ordered(int64_t n) const { return geo->kv > 1 && geo->kv <= 32 && n > kOrderRows; }

  void tables(const Tensor& oi, const Side& f, const Side& b) {
    check(spc_rulebook_tables(&geo->g, ints(indices), n_in, n_out, workspace.data_ptr(), workspace.numel(), ints(oi), ints(f.cm),
                              ints(f.rm), ints(f.order), ints(b.cm), ints(b.rm), ints(b.order), stream_of(indices)));
  }
  Side new_side(int64_t n, bool colmajor, bool order = true) const {
    Side s;
    s.rm = make(n, geo->kvp);
    if (colmajor) s.cm = make(geo->kv, n);
    if (order && ordered(n)) s.order = at::empty({n}, indices.options());
    return s;
  }
  // The side whose rows are the output rows (of the layer, or of its inverse with `input`); with the row order, where
  // such a rulebook has one, if `order`.
  Side side(bool input, bool colmajor, bool order) {
    if (input && subm()) throw Failure(SPC_ERR_INVALID_ARGUMENT, "a submanifold rulebook has one side");
    c10::cuda::CUDAGuard guard(indices.device());
    // A capture records its kernels and does not run them: it waits for nothing (what came before a capture is
    // done when the graph runs), and tables that it makes are its own.
    const bool capturing = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    std::lock_guard<std::mutex> hold(lock);
    captured = captured || capturing;
    Side& kept = input ? bwd : fwd;
    Late& late = input ? late_bwd : late_fwd;
    const bool no_cm = colmajor && !kept.cm.defined();
    const bool no_order = order && subm() && !kept.order.defined() && ordered(n_out) && n_out <= kLateOrderRows;
    const bool missing = !kept.rm.defined() || no_cm || no_order;
    if (!missing && !late.stream) return kept;
    const auto now = c10::cuda::getCurrentCUDAStream();
    Side s = kept;
    if (late.stream && *late.stream != now && !capturing) {
      late.made.block(now);
      for (const Tensor& t : {s.rm, s.cm, s.order})
        if (t.defined()) t.record_stream(now);
    }
    if (!missing) return s;
    if (!s.rm.defined()) {
      for (const Tensor& t : {indices, workspace}) t.record_stream(now);
      s = new_side(n_in, colmajor);
      tables(Tensor(), Side(), s);
    } else {
      const int64_t n = s.rm.size(0);
      s.rm.record_stream(now);
      if (no_cm) {
        s.cm = make(geo->kv, n);
        check(spc_rowmajor_to_pairs(ints(s.rm), geo->kv, n, ints(s.cm), now.stream()));
      }
      if (no_order) {
        s.order = at::empty({n}, indices.options());
        const Tensor keys = at::empty_like(s.order);
        check(spc_rowmajor_order(&geo->g, ints(s.rm), n, ints(s.order), reinterpret_cast<uint32_t*>(ints(keys)), now.stream()));
      }
    }
    if (capturing) return s;
    kept = s;
    late.made.record(now);
    late.stream = now;
    if (bwd.rm.defined() && !captured) workspace = Tensor();  // nothing is made from it any more
    return s;
  }
  std::vector<Tensor> parts() const {
    std::lock_guard<std::mutex> hold(lock);
    std::vector<Tensor> all;
    for (const Tensor& t : {indices, out_indices, workspace, fwd.rm, fwd.cm, fwd.order, bwd.rm, bwd.cm, bwd.order})
      if (t.defined()) all.push_back(t);
    return all;
  }
};
using Book = std::shared_ptr<Rulebook>;

// Returns a rulebook with n_out == 0 where no point is left.
Book build_rulebook(const std::shared_ptr<Geometry>& geo, Tensor indices, bool input_side, bool colmajor, bool order) {
  pybind11::gil_scoped_release release;
  c10::cuda::CUDAGuard guard(indices.device());
  auto rb = std::make_shared<Rulebook>();
  rb->geo = geo;
  rb->indices = indices = indices.contiguous();
  rb->n_in = indices.size(0);
  const size_t bytes = spc_rulebook_workspace_bytes(&geo->g, rb->n_in);
  if (bytes == 0) throw pybind11::value_error("rulebook geometry rejected by libspconv_b200");
  rb->workspace = at::empty({static_cast<int64_t>(bytes)}, indices.options().dtype(at::kByte));
  check(spc_rulebook_prepare(&geo->g, ints(indices), rb->n_in, rb->workspace.data_ptr(), bytes, &rb->n_out, stream_of(indices)));
  if (rb->n_out == 0) return rb;
  Rulebook::Side f = rb->new_side(rb->n_out, colmajor, order), b;
  rb->out_indices = geo->subm ? indices : rb->make(rb->n_out, geo->g.ndim + 1);
  if (input_side && !geo->subm) b = rb->new_side(rb->n_in, false, order);
  rb->tables(geo->subm ? Tensor() : rb->out_indices, f, b);
  rb->fwd = f;
  rb->bwd = b;
  if (geo->subm || b.rm.defined()) rb->workspace = Tensor();
  return rb;
}

void record_stream(const Book& rb, const Tensor& like) {
  const auto st = c10::cuda::getCurrentCUDAStream(like.device().index());
  for (const Tensor& t : rb->parts()) t.record_stream(st);
}

// ---- fp32 operands for the tensor cores ----------------------------------------------------------------------

// How fp32 operands are multiplied: on the CUDA cores, or prepared as TF32 numbers (rounded once, or split in
// two for IEEE accuracy, where the reduction is short enough for the tensor cores' accumulator).
struct Fp32Plan {
  bool tensor = false;
  int rows_mode = 0, weight_mode = 0, mult = 1;
};
// An IEEE fp32 layer on the kernel for few rows, which reads no row order.
bool few_rows(int64_t rows, int n_dim, int r_dim, int kv, bool tf32) { return !tf32 && spc_conv_small(rows, n_dim, r_dim, kv) != 0; }
Fp32Plan fp32_plan(int64_t rows, int n_dim, int r_dim, int kv, bool tf32, int split_most) {
  Fp32Plan p;
  if (few_rows(rows, n_dim, r_dim, kv, tf32)) return p;
  if (n_dim % 16 || n_dim < 16 || n_dim > 256 || r_dim % 8) return p;
  if (tf32) {
    p.tensor = true;
    p.rows_mode = p.weight_mode = SPC_TF32_ROUND;
  } else if (kv * r_dim <= split_most) {
    p.tensor = true;
    p.rows_mode = SPC_TF32_SPLIT_A;
    p.weight_mode = SPC_TF32_SPLIT_B;
    p.mult = 3;
  }
  return p;
}
// The prepared copies of a call's operands, in one block and one launch; they live as long as the call.  (Kept from
// one call for the next, a copy of the weight would have to notice every way in which a weight can change, those that
// pass its version counter by among them, and outlive captures.)
// transposed: 0 as it is, 1 as the input gradient reads it, 2 with the offsets reversed as well.
struct Prepared {
  Tensor block;
  const float *rows, *weight;
};
Prepared prepared(const Tensor& x, const Tensor& w, int transposed, const Fp32Plan& p) {
  const int64_t k_out = w.size(0), c_in = w.size(w.dim() - 1), kv = w.numel() / (k_out * c_in);
  const int64_t rows = p.mult * x.numel();  // (a multiple of eight: the weight's part starts at a 32-byte boundary)
  Prepared out{at::empty({rows + p.mult * w.numel()}, x.options()), nullptr, nullptr};
  float* at = out.block.data_ptr<float>();
  check(spc_tf32_prepare_operands(x.data_ptr<float>(), at, x.size(0), x.size(1), p.rows_mode, w.data_ptr<float>(), at + rows, k_out, kv, c_in,
                                  transposed, p.weight_mode, stream_of(x)));
  out.rows = at;
  out.weight = at + rows;
  return out;
}

// ---- convolution -------------------------------------------------------------------------------------------------

struct ConvOptions {
  bool inverse = false;  // the rulebook of a strided layer run backwards
  bool tf32 = false;
  int split_most = 0;    // longest reduction that the split fp32 operands may have
};

Tensor conv_forward_raw(const Tensor& features, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Book& rb,
                        const ConvOptions& o, at::ScalarType out_type, Tensor scale, Tensor shift, int act, double alpha) {
  on_one_device({&features, &weight, &bias, &residual, &scale, &shift, &rb->indices});
  c10::cuda::CUDAGuard guard(features.device());
  Tensor x = operand(features), w = operand(weight.scalar_type() == x.scalar_type() ? weight : weight.to(x.scalar_type()));
  int64_t k_out = w.size(0), c_in = w.size(w.dim() - 1), kv = rb->geo->kv;
  const int64_t n_in = o.inverse ? rb->n_out : rb->n_in, n_out = o.inverse ? rb->n_in : rb->n_out;
  if (x.size(0) != n_in || x.size(1) != c_in || w.numel() != k_out * kv * c_in)
    throw pybind11::value_error("features do not match the rulebook or the weight of the layer");
  Tensor b = bias;
  if (b.defined() && b.scalar_type() != x.scalar_type()) {
    if (!shift.defined() && b.scalar_type() == at::kFloat) {
      shift = b.contiguous();  // added in fp32
      b = Tensor();
    } else {
      b = b.to(x.scalar_type());
    }
  }
  if (b.defined()) b = b.contiguous();
  Tensor r = residual.defined() ? operand(residual) : residual;
  Tensor out = at::empty({n_out, k_out}, x.options().dtype(out_type));
  const void *from = x.data_ptr(), *weights = w.data_ptr();
  Prepared copies;
  int precision = x.scalar_type() == at::kFloat && o.tf32 ? SPC_PREC_TF32 : SPC_PREC_IEEE;
  if (x.scalar_type() == at::kFloat && out_type == at::kFloat) {
    const Fp32Plan plan = fp32_plan(n_out, k_out, c_in, kv, o.tf32, o.split_most);
    if (plan.tensor) {
      copies = prepared(x, w, 0, plan);
      from = copies.rows;
      weights = copies.weight;
      c_in *= plan.mult;
      precision = SPC_PREC_TF32;
    }
  }
  const int type = code_of(x.scalar_type()), out_code = code_of(out_type);
  const bool colmajor = spc_conv_forward_needs_colmajor(c_in, k_out, kv, type, out_code, precision, SPC_GEMM_AUTO);
  const Rulebook::Side t = rb->side(o.inverse, colmajor, !(type == SPC_F32 && out_code == SPC_F32 && few_rows(n_out, k_out, c_in, kv, o.tf32)));
  check(spc_conv_forward_residual(from, weights, data(b), ints(t.cm), ints(t.rm), ints(t.order), out.data_ptr(), n_in, n_out,
                                  c_in, k_out, kv, type, out_code, precision, SPC_GEMM_AUTO,
                                  scale.defined() ? scale.data_ptr<float>() : nullptr, shift.defined() ? shift.data_ptr<float>() : nullptr,
                                  act, static_cast<float>(alpha), data(r), stream_of(x)));
  return out;
}

Tensor conv_backward_input_raw(const Tensor& grad, const Tensor& weight, const Book& rb, const ConvOptions& o) {
  const int64_t k_out = weight.size(0), c_in = weight.size(weight.dim() - 1), kv = rb->geo->kv;
  const int64_t n_grad = o.inverse ? rb->n_in : rb->n_out, n_in = o.inverse ? rb->n_out : rb->n_in;
  Tensor w = operand(weight.scalar_type() == grad.scalar_type() ? weight : weight.to(grad.scalar_type()));
  Tensor din = at::empty({n_in, c_in}, grad.options());
  // a submanifold layer's input side is its output side with the offsets reversed
  const bool reversed = rb->subm(), input = !reversed && !o.inverse;
  const int type = code_of(grad.scalar_type());
  const int precision = type == SPC_F32 && o.tf32 ? SPC_PREC_TF32 : SPC_PREC_IEEE;
  const Fp32Plan plan = type == SPC_F32 ? fp32_plan(n_in, c_in, k_out, kv, o.tf32, o.split_most) : Fp32Plan();
  if (plan.tensor) {
    // as a forward convolution of grad with the transposed weight
    const Prepared copies = prepared(grad, w, reversed ? 2 : 1, plan);
    const bool colmajor = spc_conv_forward_needs_colmajor(plan.mult * k_out, c_in, kv, type, type, SPC_PREC_TF32, SPC_GEMM_AUTO);
    const Rulebook::Side t = rb->side(input, colmajor, true);
    check(spc_conv_forward(copies.rows, copies.weight, nullptr, ints(t.cm), ints(t.rm), ints(t.order), din.data_ptr(), n_grad, n_in,
                           plan.mult * k_out, c_in, kv, type, type, SPC_PREC_TF32, SPC_GEMM_AUTO, nullptr, nullptr, SPC_ACT_NONE, 0.f,
                           stream_of(grad)));
    return din;
  }
  const bool colmajor = spc_conv_backward_input_needs_colmajor(c_in, k_out, kv, type, precision, SPC_GEMM_AUTO);
  const Rulebook::Side t = rb->side(input, colmajor, !(type == SPC_F32 && few_rows(n_in, c_in, k_out, kv, o.tf32)));
  check(spc_conv_backward_input_tables(grad.data_ptr(), w.data_ptr(), ints(t.cm), ints(t.rm), ints(t.order), din.data_ptr(), n_in, n_grad,
                                       c_in, k_out, kv, reversed, type, precision, SPC_GEMM_AUTO, stream_of(grad)));
  return din;
}

Tensor conv_backward_weight_raw(const Tensor& features, const Tensor& grad, at::IntArrayRef sizes, const Book& rb, const ConvOptions& o) {
  const int64_t k_out = sizes[0], c_in = sizes[sizes.size() - 1], kv = rb->geo->kv;
  Tensor dw = at::empty(sizes, grad.options());
  Tensor x = operand(features.scalar_type() == grad.scalar_type() ? features : features.to(grad.scalar_type()));
  const Rulebook::Side t = rb->side(o.inverse, true, false);
  const int64_t n_out = grad.size(0);
  const size_t bytes = spc_conv_backward_weight_workspace_bytes(n_out, c_in, k_out, kv);
  Tensor ws = at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 16))}, grad.options().dtype(at::kByte));
  const int type = code_of(grad.scalar_type());
  check(spc_conv_backward_weight(x.data_ptr(), grad.data_ptr(), ints(t.cm), dw.data_ptr(), ws.data_ptr(), ws.numel(), x.size(0), n_out,
                                 c_in, k_out, kv, type, type == SPC_F32 && o.tf32 ? SPC_PREC_TF32 : SPC_PREC_IEEE, SPC_GEMM_AUTO,
                                 stream_of(grad)));
  return dw;
}

Tensor column_sums(const Tensor& x, at::ScalarType out_type) {
  const int64_t rows = x.size(0), cols = x.size(1);
  Tensor out = at::empty({cols}, x.options().dtype(out_type));
  Tensor ws = at::empty({static_cast<int64_t>(std::max<size_t>(spc_column_sums_workspace_bytes(rows, cols), 16))}, x.options().dtype(at::kByte));
  check(spc_column_sums(x.data_ptr(), rows, cols, code_of(x.scalar_type()), out.data_ptr(), code_of(out_type), ws.data_ptr(), ws.numel(),
                        stream_of(x)));
  return out;
}

// Backward of these layers cannot be differentiated again: with create_graph the gradients carry an error.
variable_list once_differentiable(variable_list&& out, const variable_list& grads, bool create_graph) {
  bool any = false;
  for (const Tensor& g : grads) any = any || (g.defined() && g.requires_grad());
  if (!create_graph || !any) return std::move(out);
  at::AutoGradMode grad(true);
  auto error = std::shared_ptr<torch::autograd::DelayedError>(
      new torch::autograd::DelayedError("trying to differentiate twice a function that was marked with @once_differentiable", out.size()),
      torch::autograd::deleteNode);
  for (Tensor& t : out)
    if (t.defined()) t = t.detach().set_requires_grad(true);
  return (*error)(std::move(out));
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// These layers have no forward-mode derivative (nor had the autograd functions whose place their nodes take).
void refuse_forward_mode(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->defined() && t->_fw_grad(0).defined()) {
      PyErr_SetString(PyExc_NotImplementedError, "sparse convolution and pooling layers do not support forward mode AD");
      throw pybind11::error_already_set();
    }
}

// Inside autocast these layers compute in fp16 whatever its type, as the reference's functions do.
Tensor cast_for_autocast(const Tensor& t) {
  if (!at::autocast::is_autocast_enabled(at::kCUDA) || !t.defined() || !t.is_floating_point() || t.scalar_type() == at::kDouble) return t;
  return t.to(at::kHalf);
}

struct ConvBackward : public torch::autograd::Node {
  SavedVariable features_, weight_;
  Book rb;
  ConvOptions options;
  bool bias = false, residual = false;
  at::ScalarType bias_type = at::kFloat;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> hold(mutex_);
    variable_list out(4);
    if (!grads[0].defined()) return out;
    const Tensor weight = weight_.unpack();
    Tensor features;
    if (task_should_compute_output(1)) features = features_.unpack();
    const bool create_graph = at::GradMode::is_enabled();
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(grads[0].device());
    Tensor grad = operand(grads[0]);
    if (bias && task_should_compute_output(2)) out[2] = bias_type == at::kDouble ? column_sums(grad, at::kFloat).to(at::kDouble) : column_sums(grad, bias_type);
    if (task_should_compute_output(0)) out[0] = conv_backward_input_raw(grad, weight, rb, options);
    if (task_should_compute_output(1)) out[1] = conv_backward_weight_raw(features, grad, weight.sizes(), rb, options);
    if (residual && task_should_compute_output(3)) out[3] = grads[0];
    return once_differentiable(std::move(out), grads, create_graph);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    features_.reset_data();
    weight_.reset_data();
    rb.reset();
  }
  std::string name() const override { return "SparseImplicitGemmFunctionBackward"; }
};

// A convolution in training: out = gather-GEMM (+ bias) (+ residual), with its place in the autograd graph.
Tensor conv_train(const Tensor& features, const Tensor& weight, const c10::optional<Tensor>& bias_opt, const c10::optional<Tensor>& residual_opt,
                  const Book& rb, bool inverse, bool tf32, int split_most) {
  const Tensor bias = bias_opt.value_or(Tensor()), residual = residual_opt.value_or(Tensor());
  refuse_forward_mode({&features, &weight, &bias, &residual});
  pybind11::gil_scoped_release release;
  const bool grad = wants_grad({&features, &weight, &bias, &residual});
  ConvOptions o{inverse, tf32, split_most};
  Tensor x, w, out;
  {
    at::NoGradGuard no_grad;
    x = cast_for_autocast(features).contiguous();
    w = cast_for_autocast(weight).contiguous();
    out = conv_forward_raw(x, w, bias, residual, rb, o, x.scalar_type(), Tensor(), Tensor(), SPC_ACT_NONE, 0.0);
  }
  if (!grad) return out;
  auto node = std::shared_ptr<ConvBackward>(new ConvBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(features, weight, bias, residual));
  node->features_ = SavedVariable(x, false);
  node->weight_ = SavedVariable(w, false);
  node->rb = rb;
  node->options = o;
  node->bias = bias.defined();
  node->residual = residual.defined();
  if (bias.defined()) node->bias_type = bias.scalar_type();
  torch::autograd::set_history(out, node);
  return out;
}

Tensor conv_eval(const Tensor& features, const Tensor& weight, const c10::optional<Tensor>& bias, const Book& rb, bool inverse, bool tf32,
                 int split_most, const c10::optional<Tensor>& scale, const c10::optional<Tensor>& shift, int act, double alpha) {
  pybind11::gil_scoped_release release;
  at::NoGradGuard no_grad;
  return conv_forward_raw(features, weight, bias.value_or(Tensor()), Tensor(), rb, ConvOptions{inverse, tf32, split_most},
                          weight.scalar_type(), scale.value_or(Tensor()), shift.value_or(Tensor()), act, alpha);
}

// ---- normalisation and activation -----------------------------------------------------------------------------------

Tensor norm_scratch(const Tensor& x, int type) {
  const size_t bytes = spc_norm_act_workspace_bytes(x.size(0), static_cast<int>(x.size(1)), type);
  return at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 16))}, x.options().dtype(at::kByte));
}
float* floats(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

struct NormActBackward : public torch::autograd::Node {
  SavedVariable x_, weight_, bias_;
  Tensor mean, invstd;  // (of the forward pass; nobody else has them)
  int act = 0;
  double eps = 0.0;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> hold(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const Tensor saved_x = x_.unpack(), saved_weight = weight_.unpack(), saved_bias = bias_.unpack();
    TORCH_CHECK(mean.defined(), torch::autograd::ERR_BACKWARD_TWICE);
    c10::cuda::CUDAGuard guard(grads[0].device());
    if (at::GradMode::is_enabled()) {
      // Gradients that are to be differentiated themselves: those of torch's functions of the same operands.
      const Tensor z = at::batch_norm(saved_x, saved_weight, saved_bias, Tensor(), Tensor(), true, 0.0, eps, false);
      const Tensor y = act == SPC_NORM_SILU ? at::silu(z) : act == SPC_NORM_RELU ? at::relu(z) : z;
      variable_list wanted;
      std::vector<int> at;
      const Tensor operands[3] = {saved_x, saved_weight, saved_bias};
      for (int i = 0; i < 3; ++i)
        if (task_should_compute_output(i) && operands[i].defined()) {
          wanted.push_back(operands[i]);
          at.push_back(i);
        }
      if (wanted.empty()) return out;
      const variable_list found = torch::autograd::grad({y}, wanted, {grads[0]}, true, true, true);
      for (size_t i = 0; i < at.size(); ++i) out[at[i]] = found[i];
      return out;
    }
    Tensor dy = grads[0].scalar_type() == saved_x.scalar_type() ? grads[0] : grads[0].to(saved_x.scalar_type());
    dy = operand(dy);
    // (a hook of saved tensors may give back other strides than it was given)
    const Tensor x = operand(saved_x);
    const Tensor weight = saved_weight.defined() ? saved_weight.contiguous() : saved_weight;
    const Tensor bias = saved_bias.defined() ? saved_bias.contiguous() : saved_bias;
    Tensor dx, dweight, dbias;
    if (task_should_compute_output(0)) dx = at::empty_like(x);
    if (weight.defined() && task_should_compute_output(1)) dweight = at::empty_like(weight);
    if (bias.defined() && task_should_compute_output(2)) dbias = at::empty_like(bias);
    const int type = code_of(x.scalar_type());
    const Tensor ws = norm_scratch(x, type);
    check(spc_norm_act_backward(x.data_ptr(), dy.data_ptr(), floats(weight), floats(bias), floats(mean), floats(invstd), act, data(dx),
                                floats(dweight), floats(dbias), ws.data_ptr(), ws.numel(), x.size(0), x.size(1), type, stream_of(x)));
    out[0] = dx;
    out[1] = dweight;
    out[2] = dbias;
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    x_.reset_data();
    weight_.reset_data();
    bias_.reset_data();
    mean.reset();
    invstd.reset();
  }
  std::string name() const override { return "SparseBatchNormActBackward"; }
};

bool wide_floats(const Tensor& t, int64_t n, const Tensor& like) {
  return t.scalar_type() == at::kFloat && t.dim() == 1 && t.size(0) == n && t.is_contiguous() && t.device() == like.device() &&
         t.layout() == at::kStrided && !t._fw_grad(0).defined();
}

// BatchNorm1d in training and the activation after it; nothing where the operands are not what the kernels take (the
// modules run then, and refuse what they refuse).
c10::optional<Tensor> norm_act_train(const Tensor& x, const c10::optional<Tensor>& weight_opt, const c10::optional<Tensor>& bias_opt,
                                     const Tensor& running_mean, const Tensor& running_var, const Tensor& batches, double momentum, double eps,
                                     int act) {
  const Tensor weight = weight_opt.value_or(Tensor()), bias = bias_opt.value_or(Tensor());
  const auto type = x.scalar_type();
  if ((type != at::kHalf && type != at::kBFloat16 && type != at::kFloat) || !x.is_cuda() || x.layout() != at::kStrided || x.dim() != 2 ||
      !x.is_contiguous() || (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) != 0 || x._fw_grad(0).defined() ||
      weight.defined() != bias.defined())
    return c10::nullopt;
  const int64_t rows = x.size(0), cols = x.size(1);
  if (cols > 4096 || spc_norm_act_workspace_bytes(rows, static_cast<int>(cols), code_of(type)) == 0) return c10::nullopt;
  for (const Tensor* t : {&weight, &bias, &running_mean, &running_var})
    if (t->defined() && !wide_floats(*t, cols, x)) return c10::nullopt;
  if (batches.scalar_type() != at::kLong || batches.numel() != 1 || batches.device() != x.device()) return c10::nullopt;
  pybind11::gil_scoped_release release;
  const bool grad = wants_grad({&x, &weight, &bias});
  Tensor y, mean, invstd;
  {
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(x.device());
    y = at::empty_like(x);
    mean = at::empty({cols}, x.options().dtype(at::kFloat));
    invstd = at::empty_like(mean);
    const Tensor ws = norm_scratch(x, code_of(type));
    check(spc_norm_act_forward(x.data_ptr(), floats(weight), floats(bias), floats(running_mean), floats(running_var),
                               batches.data_ptr<int64_t>(), static_cast<float>(momentum), static_cast<float>(eps), act, y.data_ptr(),
                               floats(mean), floats(invstd), ws.data_ptr(), ws.numel(), rows, static_cast<int>(cols), code_of(type),
                               stream_of(x)));
    batches.unsafeGetTensorImpl()->bump_version();  // (as its own increment does)
  }
  if (!grad) return y;
  auto node = std::shared_ptr<NormActBackward>(new NormActBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(x, weight, bias));
  node->x_ = SavedVariable(x, false);
  node->weight_ = SavedVariable(weight, false);
  node->bias_ = SavedVariable(bias, false);
  node->mean = mean;
  node->invstd = invstd;
  node->act = act;
  node->eps = eps;
  torch::autograd::set_history(y, node);
  return y;
}

// Scale and shift of evaluation-mode normalisations (mean, variance, weight, bias, eps, channels): a block for them, where in it
// each pair lies, and the argument of spc_fold_norms, which fills it; nothing where a tensor is not what the kernel takes.
using Norm = std::tuple<Tensor, Tensor, c10::optional<Tensor>, c10::optional<Tensor>, double, int64_t>;
using Places = std::vector<std::pair<int64_t, int64_t>>;
c10::optional<std::tuple<Tensor, Places, std::vector<spc_norm_fold>>> place_folds(const std::vector<Norm>& norms, const Tensor& like) {
  std::vector<spc_norm_fold> folds(norms.size());
  Places places(norms.size());
  int64_t total = 0;
  for (size_t i = 0; i < norms.size(); ++i) {
    const auto& [mean, var, weight, bias, eps, c] = norms[i];
    const Tensor none, *ts[4] = {&mean, &var, weight ? &*weight : &none, bias ? &*bias : &none};
    const void* at[4];
    for (int t = 0; t < 4; ++t) {
      at[t] = nullptr;
      folds[i].types[t] = SPC_F32;
      if (!ts[t]->defined()) continue;
      const auto type = ts[t]->scalar_type();
      if (ts[t]->layout() != at::kStrided || ts[t]->device() != like.device() || ts[t]->dim() != 1 || ts[t]->numel() != c || c == 0 ||
          !ts[t]->is_contiguous() || (type != at::kHalf && type != at::kBFloat16 && type != at::kFloat))
        return c10::nullopt;
      at[t] = ts[t]->const_data_ptr();
      folds[i].types[t] = code_of(type);
    }
    folds[i].mean = at[0];
    folds[i].var = at[1];
    folds[i].weight = at[2];
    folds[i].bias = at[3];
    folds[i].channels = static_cast<int32_t>(c);
    folds[i].eps = static_cast<float>(eps);
    const int64_t room = (c + 3) & ~int64_t{3};
    places[i] = {total, total + room};
    total += 2 * room;
  }
  at::NoGradGuard no_grad;
  c10::cuda::CUDAGuard guard(like.device());
  Tensor block = at::empty({total}, like.options().dtype(at::kFloat));
  for (size_t i = 0; i < norms.size(); ++i) {
    folds[i].scale = block.data_ptr<float>() + places[i].first;
    folds[i].shift = block.data_ptr<float>() + places[i].second;
  }
  return std::make_tuple(block, std::move(places), std::move(folds));
}
c10::optional<std::tuple<Tensor, Places, pybind11::bytes>> norm_folds(const std::vector<Norm>& norms, const Tensor& like) {
  auto placed = place_folds(norms, like);
  if (!placed) return c10::nullopt;
  auto& [block, places, folds] = *placed;
  return std::make_tuple(block, places, pybind11::bytes(reinterpret_cast<const char*>(folds.data()), folds.size() * sizeof(spc_norm_fold)));
}
// Scale and shift of one of them, made on the current stream.
c10::optional<std::pair<Tensor, Tensor>> fold_norm(const Tensor& mean, const Tensor& var, const c10::optional<Tensor>& weight,
                                                   const c10::optional<Tensor>& bias, double eps, int64_t c, const Tensor& like) {
  const auto placed = place_folds({Norm{mean, var, weight, bias, eps, c}}, like);
  if (!placed) return c10::nullopt;
  const auto& [block, places, folds] = *placed;
  at::NoGradGuard no_grad;
  c10::cuda::CUDAGuard guard(like.device());
  check(spc_fold_norms(folds.data(), 1, stream_of(like)));
  return std::make_pair(block.narrow(0, places[0].first, c), block.narrow(0, places[0].second, c));
}

// ---- pooling -------------------------------------------------------------------------------------------------------

// Bytes of gathered rows from which on the gradient of an average works on the input rows in the order of the
// outputs they read.  Input rows come as the user has them, outputs in cell order: up to about the size of the L2
// (126 MB) that does not matter, beyond it every gather of an unordered row is a miss (27 outputs of 512 bytes each,
// 300 k rows: 741 -> 439 us, the order itself 28 us in four launches).  The maximum's gradient, which reads few
// outputs a row and its own row besides, gains nothing (213 against 227 us).
constexpr size_t kPoolOrderBytes = size_t{96} << 20;

Tensor pool_rows(int op, const Tensor& src, const Tensor& own, const Tensor& ref, const Book& rb, bool input, const Tensor& aux_in,
                 const Tensor& aux_out) {
  const int64_t c = src.size(1);
  const bool flip = rb->subm() && input;  // (a pool over a submanifold neighbourhood: the table of the other side)
  const Rulebook::Side t = rb->side(input && !flip, false, false);
  const int64_t n = t.rm.size(0);
  Tensor out = at::empty({n, c}, src.options());
  if (c == 0) return out;
  Tensor order;
  if (op == SPC_POOL_AVG_BACKWARD && n > 0 && src.nbytes() >= kPoolOrderBytes) {
    order = at::empty({n}, rb->indices.options());
    Tensor scratch = at::empty({static_cast<int64_t>(spc_pool_row_order_workspace_bytes(n))}, rb->indices.options().dtype(at::kByte));
    check(spc_pool_row_order(ints(t.rm), rb->geo->kvp, rb->geo->kv, n, src.size(0), ints(order), scratch.data_ptr(), scratch.numel(),
                             stream_of(src)));
  }
  check(spc_pool(op, src.data_ptr(), data(own), data(ref), ints(t.rm), rb->geo->kvp, ints(order), ints(aux_in), out.data_ptr(), ints(aux_out), n, c,
                 rb->geo->kv, code_of(src.scalar_type()), stream_of(src)));
  return out;
}

struct PoolBackward : public torch::autograd::Node {
  SavedVariable features_, out_, count_;
  Book rb;
  bool average = false;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> hold(mutex_);
    variable_list result(1);
    if (!grads[0].defined() || !task_should_compute_output(0)) return result;
    Tensor features, out, count;
    if (average) {
      count = count_.unpack().contiguous();  // (a hook of saved tensors may give back other strides than it was given)
    } else {
      features = features_.unpack().contiguous();
      out = out_.unpack(shared_from_this()).contiguous();
    }
    const bool create_graph = at::GradMode::is_enabled();
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(grads[0].device());
    Tensor grad = grads[0].contiguous();
    if (average) {
      result[0] = pool_rows(SPC_POOL_AVG_BACKWARD, grad, Tensor(), Tensor(), rb, true, count, Tensor());
    } else {
      if (grad.scalar_type() != features.scalar_type()) grad = grad.to(features.scalar_type());
      result[0] = pool_rows(SPC_POOL_MAX_BACKWARD, grad, features, out, rb, true, Tensor(), Tensor());
    }
    return once_differentiable(std::move(result), grads, create_graph);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    features_.reset_data();
    out_.reset_data();
    count_.reset_data();
    rb.reset();
  }
  std::string name() const override {
    return average ? "SparseAvgPoolImplicitGemmFunctionBackward" : "SparseMaxPoolImplicitGemmFunctionBackward";
  }
};

Tensor pool(const Tensor& features, const Book& rb, bool average) {
  refuse_forward_mode({&features});
  pybind11::gil_scoped_release release;
  const bool grad = wants_grad({&features});
  Tensor x, out, count;
  {
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(features.device());
    x = cast_for_autocast(features).contiguous();
    on_one_device({&x, &rb->indices});
    if (x.size(0) != rb->n_in) throw pybind11::value_error("features do not match the rulebook of the layer");
    if (average) count = at::empty({rb->n_out}, rb->indices.options());
    out = pool_rows(average ? SPC_POOL_AVG_FORWARD : SPC_POOL_MAX_FORWARD, x, Tensor(), Tensor(), rb, false, Tensor(), count);
  }
  if (!grad) return out;
  auto node = std::shared_ptr<PoolBackward>(new PoolBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(features));
  node->rb = rb;
  node->average = average;
  torch::autograd::set_history(out, node);
  if (average) {
    node->count_ = SavedVariable(count, false);
  } else {
    node->features_ = SavedVariable(x, false);
    node->out_ = SavedVariable(out, true);
  }
  return out;
}

// ---- voxelisation ----------------------------------------------------------------------------------------------------

// (voxels, indices, num_per_voxel of the voxels found, pc_voxel_id); the persistent buffers hold the same.
std::tuple<Tensor, Tensor, Tensor, Tensor> voxelize(const Tensor& points, const Tensor& voxels, const Tensor& indices, const Tensor& num,
                                                    const std::vector<float>& cmin, const std::vector<float>& vsize,
                                                    const std::vector<int32_t>& grid, bool clear, bool empty_mean) {
  pybind11::gil_scoped_release release;
  at::NoGradGuard no_grad;
  on_one_device({&points, &voxels, &indices, &num});
  c10::cuda::CUDAGuard guard(points.device());
  const Tensor pc = points.contiguous();
  const int64_t n = pc.size(0), most = voxels.size(0);
  const int nd = static_cast<int>(cmin.size()), slots = static_cast<int>(voxels.size(1)), f = static_cast<int>(voxels.size(2));
  const int stride = static_cast<int>(pc.size(1));
  const size_t bytes = spc_voxelize_workspace_bytes(n, most, slots);
  if (bytes == 0) throw Failure(SPC_ERR_SIZE_LIMIT, "voxelize: sizes out of range");
  Tensor id = at::empty({n}, pc.options().dtype(at::kLong)), ws = at::empty({static_cast<int64_t>(bytes)}, pc.options().dtype(at::kByte));
  void* st = stream_of(pc);
  int64_t found = 0;
  int sorted = 0;
  float* at_points = n ? pc.data_ptr<float>() : nullptr;
  int64_t* at_id = n ? id.data_ptr<int64_t>() : nullptr;
  check(spc_voxelize_number(at_points, n, stride, nd, f, cmin.data(), vsize.data(), grid.data(), most, slots, ws.data_ptr(), bytes,
                            ints(indices), ints(num), at_id, &found, &sorted, st));
  // without the clear the copy shows what the slots held before
  const bool together = clear;
  Tensor v, i, c;
  if (together) {
    v = at::empty({found, slots, f}, voxels.options());
    i = at::empty({found, nd}, indices.options());
    c = at::empty({found}, num.options());
  }
  check(spc_voxelize_store(at_points, n, stride, nd, f, most, slots, clear, empty_mean, ws.data_ptr(), bytes, found, sorted, ints(indices),
                           ints(num), at_id, voxels.data_ptr<float>(), together ? v.data_ptr<float>() : nullptr,
                           together ? ints(i) : nullptr, together ? ints(c) : nullptr, st));
  if (!together) {
    v = voxels.narrow(0, 0, found).clone();
    i = indices.narrow(0, 0, found).clone();
    c = num.narrow(0, 0, found).clone();
  }
  return {v, i, c, id};
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  namespace py = pybind11;
  static PyObject* error_type = nullptr;  // SpconvB200Error(status, message), handed over by the package
  m.def("set_error_type", [](py::object t) { error_type = t.release().ptr(); });
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const Failure& f) {
      py::object e = py::reinterpret_borrow<py::object>(error_type)(f.status, std::string(f.what()));
      PyErr_SetObject(error_type, e.ptr());
    }
  });
  py::class_<Geometry, std::shared_ptr<Geometry>>(m, "Geometry")
      .def(py::init(&make_geometry))
      .def_readonly("kv", &Geometry::kv)
      .def_readonly("subm", &Geometry::subm)
      .def_readonly("out_shape", &Geometry::out_shape);
  py::class_<Rulebook, Book>(m, "Rulebook")
      .def_readonly("n_in", &Rulebook::n_in)
      .def_readonly("n_out", &Rulebook::n_out)
      .def_readonly("geometry", &Rulebook::geo)
      .def_readonly("indices", &Rulebook::indices)
      .def_readonly("out_indices", &Rulebook::out_indices)
      .def_readonly("captured", &Rulebook::captured)
      .def("rowmajor", [](Rulebook& r, bool input) { return r.side(input, false, false).rm; }, py::call_guard<py::gil_scoped_release>())
      .def("colmajor", [](Rulebook& r, bool input) { return r.side(input, true, false).cm; }, py::call_guard<py::gil_scoped_release>());
  m.def("build_rulebook", &build_rulebook);
  m.def("record_stream", &record_stream);
  m.def("conv_train", &conv_train);
  m.def("conv_eval", &conv_eval);
  m.def("norm_act_train", &norm_act_train);
  m.def("norm_folds", &norm_folds);
  m.def("fold_norm", &fold_norm);
  // both directions of an IEEE fp32 layer run on the kernel for few rows
  m.def("small", [](int64_t rows, int c_out, int c_in, int kv) {
    return spc_conv_small(rows, c_out, c_in, kv) != 0 && spc_conv_small(rows, c_in, c_out, kv) != 0;
  });
  m.def("pool", &pool);
  m.def("voxelize", &voxelize);
}

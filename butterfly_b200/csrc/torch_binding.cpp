// Thin torch operator layer over the C ABI in include/bfly.h.
//
// Registers the operators the reference registers in csrc/butterfly.cpp:127-131
// (torch_butterfly::butterfly_multiply_fw / _bw / butterfly_multiply) with the same
// argument meaning and the same argument checks (csrc/butterfly.cpp:34-43, 72-83), plus
// native operators for the base-4 product that the reference only has as PyTorch code
// (torch_butterfly/multiply_base4.py:7-41) and torch_butterfly::cuda_version
// (csrc/version.cpp:14-23).  Everything below this file is plain pointers and sizes.
//
// CUDA tensors only: there is no CPU implementation behind these operators, and they
// raise instead of falling back when handed a CPU tensor.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/script.h>

#include <cstdlib>
#include <tuple>

#include "../../include/bfly.h"

namespace {

using torch::Tensor;

#define BFLY_CHECK_CUDA(x) \
  TORCH_CHECK((x).device().is_cuda(), #x " must be a CUDA tensor: the B200 butterfly library has no CPU path")
#define BFLY_CHECK_SAME_DEVICE(x, y) \
  TORCH_CHECK((x).device() == (y).device(), #x " and " #y " must be on the same device")
#define BFLY_CHECK_DIM(x, d) TORCH_CHECK((x).dim() == (d), #x " must have dimension " #d)

void check_status(int rc, const char* what) {
  TORCH_CHECK(rc == BFLY_OK, what, " failed: ", bfly_strerror(rc), " (status ", rc, ")");
}

int dtype_code(const Tensor& t, const char* what) {
  if (t.scalar_type() == at::kFloat) return BFLY_F32;
  if (t.scalar_type() == at::kComplexFloat) return BFLY_C64;
  TORCH_CHECK(false, what, " not implemented for '", toString(t.scalar_type()), "'");
  return -1;
}

// Borrowed tensors are never mutated; lazily-conjugated or strided views are materialised.
Tensor dense_twiddle(const Tensor& t) { return t.resolve_conj().contiguous(); }
// The kernels take complex rows from 8-byte boundaries (bfly.h).  Tensors over foreign memory may start in between; they
// are copied as floats (PyTorch's own complex copies assume the alignment too).
Tensor on_element(const Tensor& t) {
  if (!t.numel() || reinterpret_cast<uintptr_t>(t.const_data_ptr()) % t.element_size() == 0) return t;
  const bool conj = t.is_conj();
  Tensor r = at::view_as_complex(at::view_as_real(conj ? t.conj() : t).clone(at::MemoryFormat::Contiguous));
  return conj ? r.conj() : r;
}
Tensor rows_view(const Tensor& t) {
  Tensor r = on_element(t).resolve_conj();
  if (r.size(2) > 1 && r.stride(2) != 1) r = r.contiguous();
  if (r.size(2) <= 1 && r.stride(2) != 1) r = r.contiguous();
  return r;
}

// Does a call see a forward-mode tangent on this tensor?  Paths around an autograd node ask, because the node is what
// refuses tangents (no operator here has a forward-mode rule); without it they would be dropped without a word.
bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }
bool has_tangent(const c10::optional<Tensor>& t) { return t.has_value() && has_tangent(*t); }

// Shared by the plain operator and the autograd node: with `snapshots`, a buffer of bfly_fw_saving_bytes, the forward also
// writes there what the backward starts from.
Tensor fw_impl(const Tensor& twiddle, const Tensor& input, bool increasing_stride,
               c10::optional<int64_t> output_size, const Tensor* snapshots) {
  BFLY_CHECK_CUDA(twiddle); BFLY_CHECK_CUDA(input); BFLY_CHECK_SAME_DEVICE(twiddle, input);
  BFLY_CHECK_DIM(twiddle, 6); BFLY_CHECK_DIM(input, 3);
  const int64_t batch = input.size(0), nstacks = input.size(1), input_size = input.size(2);
  const int64_t nblocks = twiddle.size(1), log_n = twiddle.size(2);
  TORCH_CHECK(log_n >= 1 && log_n <= 24, "butterfly_multiply_fw: n must be a power of 2 (2 <= n <= 2^24)");
  const int64_t n = (int64_t)1 << log_n;
  TORCH_CHECK(twiddle.sizes() == torch::IntArrayRef({nstacks, nblocks, log_n, n / 2, 2, 2}),
              "twiddle must have shape (nstacks, nblocks, log_n, n / 2, 2, 2)");
  const int64_t out_size = output_size.has_value() ? output_size.value() : n;
  TORCH_CHECK(out_size <= n, "butterfly_multiply_fw: output_size must be <= n");
  TORCH_CHECK(out_size >= 0, "butterfly_multiply_fw: output_size must be >= 0");
  TORCH_CHECK(twiddle.scalar_type() == input.scalar_type(), "twiddle and input must have the same dtype");
  const int dt = dtype_code(input, "butterfly_multiply_fw_cuda");
  c10::cuda::CUDAGuard guard(input.device());
  const Tensor tw = dense_twiddle(twiddle);
  const Tensor x = rows_view(input);
  Tensor output = torch::empty({batch, nstacks, n}, input.options());
  auto stream = at::cuda::getCurrentCUDAStream();
  int rc;
  if (snapshots) {
    rc = bfly_fw_saving_ws(dt, tw.data_ptr(), x.data_ptr(), x.stride(0), x.stride(1), output.data_ptr(), (int)batch, (int)nstacks, (int)log_n,
                           (int)nblocks, (int)input_size, (int)out_size, increasing_stride, snapshots->data_ptr(), (size_t)snapshots->numel(),
                           stream.stream());
  } else {
    // optional scratch of the forward (room for the re-ordered twiddles of its fastest kernel)
    const int64_t fws = bfly_fw_workspace_bytes(dt, (int)batch, (int)nstacks, (int)log_n, (int)nblocks);
    TORCH_CHECK(fws >= 0, "butterfly_multiply_fw failed: ", bfly_strerror((int)fws));
    Tensor ws;
    if (fws > 0) ws = torch::empty({fws}, input.options().dtype(at::kByte));
    void* wp = fws > 0 ? ws.data_ptr() : nullptr;
    if (dt == BFLY_F32) {
      rc = bfly_fw_f32(tw.data_ptr<float>(), x.data_ptr<float>(), x.stride(0), x.stride(1),
                       output.data_ptr<float>(), (int)batch, (int)nstacks, (int)log_n, (int)nblocks,
                       (int)input_size, (int)out_size, increasing_stride, wp, (size_t)fws, stream.stream());
    } else {
      rc = bfly_fw_c64(tw.data_ptr(), x.data_ptr(), x.stride(0), x.stride(1), output.data_ptr(), (int)batch,
                       (int)nstacks, (int)log_n, (int)nblocks, (int)input_size, (int)out_size,
                       increasing_stride, wp, (size_t)fws, stream.stream());
    }
  }
  check_status(rc, "butterfly_multiply_fw");
  return out_size < n ? output.slice(2, 0, out_size) : output;
}

Tensor butterfly_multiply_fw(const Tensor& twiddle, const Tensor& input, bool increasing_stride,
                             c10::optional<int64_t> output_size) {
  return fw_impl(twiddle, input, increasing_stride, output_size, nullptr);
}

// `snapshots`: what the matching fw_impl call saved (then the backward skips its own forward
// pass over the first phases), or null.
std::tuple<Tensor, Tensor> bw_impl(const Tensor& twiddle, const Tensor& input, const Tensor& grad,
                                   bool increasing_stride, const Tensor* snapshots) {
  BFLY_CHECK_CUDA(twiddle); BFLY_CHECK_CUDA(input); BFLY_CHECK_CUDA(grad);
  BFLY_CHECK_SAME_DEVICE(twiddle, input); BFLY_CHECK_SAME_DEVICE(input, grad);
  BFLY_CHECK_DIM(twiddle, 6); BFLY_CHECK_DIM(input, 3); BFLY_CHECK_DIM(grad, 3);
  const int64_t batch = input.size(0), nstacks = input.size(1), input_size = input.size(2);
  const int64_t nblocks = twiddle.size(1), log_n = twiddle.size(2);
  TORCH_CHECK(log_n >= 1 && log_n <= 24, "butterfly_multiply_bw: n must be a power of 2 (2 <= n <= 2^24)");
  const int64_t n = (int64_t)1 << log_n;
  const int64_t out_size = grad.size(2);
  TORCH_CHECK(twiddle.sizes() == torch::IntArrayRef({nstacks, nblocks, log_n, n / 2, 2, 2}),
              "twiddle must have shape (nstacks, nblocks, log_n, n / 2, 2, 2)");
  TORCH_CHECK(grad.sizes() == torch::IntArrayRef({batch, nstacks, out_size}),
              "grad must have shape (batch_size, nstacks, output_size)");
  TORCH_CHECK(out_size <= n, "butterfly_multiply_bw: output_size must be <= n");
  TORCH_CHECK(twiddle.scalar_type() == input.scalar_type() && grad.scalar_type() == input.scalar_type(),
              "twiddle, input and grad must have the same dtype");
  const int dt = dtype_code(input, "butterfly_multiply_bw_cuda");
  c10::cuda::CUDAGuard guard(input.device());
  const Tensor tw = dense_twiddle(twiddle);
  const Tensor x = rows_view(input);
  const Tensor g = rows_view(grad);
  Tensor d_twiddle = torch::empty_like(tw);
  Tensor d_input = torch::empty({batch, nstacks, std::max(input_size, n)}, input.options());
  const int64_t kept = snapshots ? snapshots->numel() : 0;
  const bool saved = kept > 0;
  const int64_t ws_bytes = saved ? bfly_bw_saved_workspace_bytes(dt, (int)batch, (int)nstacks, (int)log_n, (int)nblocks)
                                 : bfly_bw_workspace_bytes(dt, (int)batch, (int)nstacks, (int)log_n, (int)nblocks);
  TORCH_CHECK(ws_bytes >= 0, "butterfly_multiply_bw failed: ", bfly_strerror((int)ws_bytes));
  Tensor ws = torch::empty({ws_bytes}, input.options().dtype(at::kByte));
  auto stream = at::cuda::getCurrentCUDAStream();
  int rc;
  if (saved) {
    rc = bfly_bw_saved_ws(dt, tw.data_ptr(), x.data_ptr(), x.stride(0), x.stride(1), g.data_ptr(), g.stride(0), g.stride(1),
                          d_twiddle.data_ptr(), d_input.data_ptr(), (int)batch, (int)nstacks, (int)log_n, (int)nblocks, (int)input_size,
                          (int)out_size, increasing_stride, snapshots->data_ptr(), (size_t)kept, ws_bytes ? ws.data_ptr() : nullptr,
                          (size_t)ws_bytes, stream.stream());
  } else if (dt == BFLY_F32) {
    rc = bfly_bw_f32(tw.data_ptr<float>(), x.data_ptr<float>(), x.stride(0), x.stride(1), g.data_ptr<float>(),
                     g.stride(0), g.stride(1), d_twiddle.data_ptr<float>(), d_input.data_ptr<float>(), (int)batch,
                     (int)nstacks, (int)log_n, (int)nblocks, (int)input_size, (int)out_size, increasing_stride,
                     ws_bytes ? ws.data_ptr() : nullptr, (size_t)ws_bytes, stream.stream());
  } else {
    rc = bfly_bw_c64(tw.data_ptr(), x.data_ptr(), x.stride(0), x.stride(1), g.data_ptr(), g.stride(0), g.stride(1),
                     d_twiddle.data_ptr(), d_input.data_ptr(), (int)batch, (int)nstacks, (int)log_n, (int)nblocks,
                     (int)input_size, (int)out_size, increasing_stride, ws_bytes ? ws.data_ptr() : nullptr,
                     (size_t)ws_bytes, stream.stream());
  }
  check_status(rc, "butterfly_multiply_bw");
  if (input_size < n) d_input = d_input.slice(2, 0, input_size);
  return std::make_tuple(d_twiddle, d_input);
}

std::tuple<Tensor, Tensor> butterfly_multiply_bw(const Tensor& twiddle, const Tensor& input, const Tensor& grad,
                                                 bool increasing_stride) {
  return bw_impl(twiddle, input, grad, increasing_stride, nullptr);
}

// The autograd nodes (the operator's and the layers') may keep the forward's phase-boundary activations for the backward (the
// reference recomputes them, csrc/butterfly.cpp:99-118): that removes one forward-sized pass from
// every training step at the price of holding (phases - 1) activation-sized buffers per call
// between forward and backward.  On by default while those buffers stay under 1 GiB per call;
// the library option "autograd_save" (environment BFLY_AUTOGRAD_SAVE at load time, or
// bfly_set_option) = 0 always recomputes, = 1 always saves.
bool autograd_saves(int64_t snapshot_bytes) {
  int v = -1;
  if (bfly_get_option("autograd_save", &v) == BFLY_OK && v >= 0) return v != 0;
  return snapshot_bytes > 0 && snapshot_bytes <= ((int64_t)1 << 30);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Same contract as the reference's autograd node (csrc/butterfly.cpp:99-118): saves
// {twiddle, input} and the direction flag, returns {d_twiddle, d_input, none, none}.
class ButterflyMultiply : public torch::autograd::Function<ButterflyMultiply> {
 public:
  // `wants_grad`: a gradient can be asked for later.  The caller decides it, because inside
  // apply() gradient mode is always off while parameters still report requires_grad: a forward
  // under torch.no_grad() must not pay for snapshots nobody will read.
  static Tensor forward(AutogradContext* ctx, Tensor twiddle, Tensor input, bool increasing_stride,
                        c10::optional<int64_t> output_size, bool wants_grad) {
    ctx->saved_data["increasing_stride"] = increasing_stride;
    int64_t ws = 0;
    if (wants_grad && twiddle.is_cuda() && input.is_cuda() && twiddle.dim() == 6 && input.dim() == 3 &&
        (input.scalar_type() == at::kFloat || input.scalar_type() == at::kComplexFloat)) {
      ctx->saved_data["options"] = bfly_option_changes();
      ws = bfly_fw_saving_bytes(input.scalar_type() == at::kFloat ? BFLY_F32 : BFLY_C64, (int)input.size(0), (int)input.size(1),
                                (int)twiddle.size(2), (int)twiddle.size(1), increasing_stride);
    }
    if (ws <= 0 || !autograd_saves(ws)) {
      ctx->save_for_backward({twiddle, input});
      return butterfly_multiply_fw(twiddle, input, increasing_stride, output_size);
    }
    const Tensor snapshots = torch::empty({ws}, input.options().dtype(at::kByte));
    Tensor out = fw_impl(twiddle, input, increasing_stride, output_size, &snapshots);
    ctx->save_for_backward({twiddle, input, snapshots});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_output) {
    auto saved = ctx->get_saved_variables();
    auto result = bw_impl(saved[0], saved[1], grad_output[0], ctx->saved_data["increasing_stride"].toBool(),
                          saved.size() > 2 && ctx->saved_data["options"].toInt() == bfly_option_changes() ? &saved[2] : nullptr);
    return {std::get<0>(result), std::get<1>(result), Tensor(), Tensor(), Tensor()};
  }
};

Tensor butterfly_multiply(const Tensor& twiddle, const Tensor& input, bool increasing_stride,
                          c10::optional<int64_t> output_size) {
  const bool wants_grad = at::GradMode::is_enabled() && (twiddle.requires_grad() || input.requires_grad());
  return ButterflyMultiply::apply(twiddle, input, increasing_stride, output_size, wants_grad);
}

// ---------------------------------------------------------------- layers
//
// A Butterfly as a layer without the PyTorch glue of the reference's modules (torch_butterfly/butterfly.py:152-169,
// butterfly_base4.py:56-72): input (..., in_size) shared by the stacks, output the first out_size columns of the
// stacks' outputs side by side, bias added in the kernels.  One autograd node whatever the input's rank: the
// reshapes, the bias and its gradient, the padding of a cut last stack and the sum over the stacks cost no operator.

struct LayerCall {
  bfly_layer_t p;
  Tensor t4, t2, x;  // dense twiddles (t4 undefined for radix 2), rows (batch, in_size)
  int64_t n, width;  // columns of a stack, of all stacks
};

Tensor rows_2d(const Tensor& t) {
  Tensor r = on_element(t);
  if (r.dim() != 2) r = r.reshape({-1, r.size(-1)});
  r = r.resolve_conj();
  return r.stride(1) == 1 ? r : r.contiguous();
}

LayerCall layer_call(const Tensor& twiddle, const Tensor& twiddle2, const Tensor& input, bool increasing_stride, int64_t out_size,
                     const char* what) {
  LayerCall c;
  const bool base4 = twiddle2.defined();
  BFLY_CHECK_CUDA(twiddle); BFLY_CHECK_CUDA(input); BFLY_CHECK_SAME_DEVICE(twiddle, input);
  BFLY_CHECK_DIM(twiddle, 6);
  TORCH_CHECK(input.dim() >= 1, what, ": input must have a last dimension");
  const int64_t nstacks = twiddle.size(0), nblocks = twiddle.size(1);
  int64_t log_n = twiddle.size(2);
  if (base4) {
    BFLY_CHECK_CUDA(twiddle2); BFLY_CHECK_SAME_DEVICE(twiddle2, input); BFLY_CHECK_DIM(twiddle2, 6);
    log_n = 2 * log_n + twiddle2.size(2);
    TORCH_CHECK(twiddle2.size(2) <= 1 && twiddle2.scalar_type() == input.scalar_type(), what, ": inconsistent twiddle2");
  }
  TORCH_CHECK(log_n >= 1 && log_n <= 24, what, ": n must be a power of 2 (2 <= n <= 2^24)");
  c.n = (int64_t)1 << log_n;
  c.width = nstacks * c.n;
  if (!base4) {
    TORCH_CHECK(twiddle.sizes() == torch::IntArrayRef({nstacks, nblocks, log_n, c.n / 2, 2, 2}),
                "twiddle must have shape (nstacks, nblocks, log_n, n / 2, 2, 2)");
  } else {
    if (log_n / 2 > 0)
      TORCH_CHECK(twiddle.sizes() == torch::IntArrayRef({nstacks, nblocks, log_n / 2, c.n / 4, 4, 4}),
                  "twiddle4 must have shape (nstacks, nblocks, log_n / 2, n / 4, 4, 4)");
    if (log_n % 2 == 1)
      TORCH_CHECK(twiddle2.sizes() == torch::IntArrayRef({nstacks, nblocks, 1, c.n / 2, 2, 2}),
                  "twiddle2 must have shape (nstacks, nblocks, 1, n / 2, 2, 2)");
  }
  TORCH_CHECK(out_size >= 0 && out_size <= c.width, what, ": out_size must be <= nstacks * n");
  TORCH_CHECK(twiddle.scalar_type() == input.scalar_type(), "twiddle and input must have the same dtype");
  c.x = rows_2d(input);
  c.p = bfly_layer_t{dtype_code(input, what), base4, (int)c.x.size(0), (int)nstacks, (int)log_n, (int)nblocks,
                     (int)c.x.size(1), (int)out_size, increasing_stride};
  if (base4) { c.t4 = dense_twiddle(twiddle); c.t2 = dense_twiddle(twiddle2); }
  else c.t2 = dense_twiddle(twiddle);
  return c;
}
const void* data_or_null(const Tensor& t) { return t.defined() && t.numel() ? t.data_ptr() : nullptr; }

// `snapshots`: when given, the activations the backward starts from are kept there if they stay under the limit
Tensor layer_fw(const Tensor& twiddle, const Tensor& twiddle2, const Tensor& input, const c10::optional<Tensor>& bias,
                bool increasing_stride, int64_t out_size, Tensor* snapshots) {
  const LayerCall c = layer_call(twiddle, twiddle2, input, increasing_stride, out_size, "butterfly_layer");
  Tensor b;
  if (bias.has_value() && bias->defined()) {
    BFLY_CHECK_CUDA((*bias)); BFLY_CHECK_SAME_DEVICE((*bias), input);
    TORCH_CHECK(bias->scalar_type() == input.scalar_type() && bias->dim() == 1 && bias->size(0) >= out_size,
                "bias must be a vector of at least out_size entries with the dtype of input");
    b = bias->resolve_conj().contiguous();
  }
  c10::cuda::CUDAGuard guard(input.device());
  Tensor output = torch::empty({c.x.size(0), c.width}, input.options());
  int64_t keep = 0, scratch = 0;
  if (snapshots) {
    keep = bfly_layer_snapshot_bytes(&c.p);
    if (keep < 0 || !autograd_saves(keep)) keep = 0;
  }
  Tensor ws;
  if (keep > 0) {
    *snapshots = torch::empty({keep}, input.options().dtype(at::kByte));
  } else if (!c.t4.defined()) {
    scratch = bfly_fw_workspace_bytes(c.p.dtype, c.p.batch, c.p.nstacks, c.p.log_n, c.p.nblocks);
    if (scratch > 0) ws = torch::empty({scratch}, input.options().dtype(at::kByte));
  }
  const int rc = bfly_layer_fw(&c.p, data_or_null(c.t2), data_or_null(c.t4), c.x.data_ptr(), c.x.stride(0), output.data_ptr(),
                               data_or_null(b), keep > 0 ? snapshots->data_ptr() : nullptr, (size_t)keep,
                               scratch > 0 ? ws.data_ptr() : nullptr, (size_t)std::max<int64_t>(scratch, 0),
                               at::cuda::getCurrentCUDAStream().stream());
  check_status(rc, "butterfly_layer");
  // A view that autograd knows as one, made inside the node, would refuse every in-place operator behind the layer
  // (ReLU(inplace=True)); below its dispatch keys the same view is a tensor of its own, and nothing else sees its base.
  at::AutoDispatchBelowADInplaceOrView no_view_tracking;
  if (input.dim() == 2) return out_size < c.width ? output.narrow(1, 0, out_size) : output;
  auto shape = input.sizes().vec();
  shape.back() = c.width;
  output = output.view(shape);
  return out_size < c.width ? output.narrow(-1, 0, out_size) : output;
}

struct LayerGrads { Tensor twiddle, twiddle2, input, bias; };
LayerGrads layer_bw(const Tensor& twiddle, const Tensor& twiddle2, const Tensor& input, const Tensor& grad, bool increasing_stride,
                    bool need_bias, const Tensor& snapshots) {
  BFLY_CHECK_CUDA(grad); BFLY_CHECK_SAME_DEVICE(input, grad);
  TORCH_CHECK(grad.scalar_type() == input.scalar_type(), "grad must have the dtype of input");
  const int64_t out_size = grad.size(-1);
  const LayerCall c = layer_call(twiddle, twiddle2, input, increasing_stride, out_size, "butterfly_layer_bw");
  c10::cuda::CUDAGuard guard(input.device());
  Tensor g = rows_2d(grad);
  TORCH_CHECK(g.size(0) == c.x.size(0), "grad must have the leading dimensions of input");
  const int64_t batch = c.x.size(0), in_size = c.x.size(1);
  LayerGrads r;
  Tensor d2 = torch::empty_like(c.t2), d4 = c.t4.defined() ? torch::empty_like(c.t4) : Tensor();
  r.twiddle = c.t4.defined() ? d4 : d2;
  if (c.t4.defined()) r.twiddle2 = d2;
  const int64_t dx_cols = c.p.nstacks > 1 ? in_size : std::max(in_size, c.n);
  Tensor dx = torch::empty({batch, dx_cols}, input.options());
  if (need_bias) r.bias = torch::empty({out_size}, input.options());
  const int64_t kept = snapshots.defined() ? snapshots.numel() : 0;
  const int64_t wsb = bfly_layer_bw_workspace_bytes(&c.p, kept > 0);
  TORCH_CHECK(wsb >= 0, "butterfly_layer_bw failed: ", bfly_strerror((int)wsb));
  Tensor ws;
  if (wsb > 0) ws = torch::empty({wsb}, input.options().dtype(at::kByte));
  const int rc = bfly_layer_bw(&c.p, data_or_null(c.t2), data_or_null(c.t4), c.x.data_ptr(), c.x.stride(0), g.data_ptr(), g.stride(0),
                               kept > 0 ? snapshots.data_ptr() : nullptr, (size_t)kept, const_cast<void*>(data_or_null(d2)),
                               const_cast<void*>(data_or_null(d4)), dx.data_ptr(), need_bias ? r.bias.data_ptr() : nullptr,
                               wsb > 0 ? ws.data_ptr() : nullptr, (size_t)wsb, at::cuda::getCurrentCUDAStream().stream());
  check_status(rc, "butterfly_layer_bw");
  if (dx_cols > in_size) dx = dx.narrow(1, 0, in_size);
  r.input = input.dim() == 2 ? dx : dx.reshape(input.sizes());
  return r;
}

class ButterflyLayer : public torch::autograd::Function<ButterflyLayer> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor twiddle, c10::optional<Tensor> twiddle2, Tensor input, c10::optional<Tensor> bias,
                        bool increasing_stride, int64_t out_size, bool wants_grad) {
    const Tensor t2 = twiddle2.has_value() ? *twiddle2 : Tensor();
    Tensor snapshots;
    if (wants_grad) ctx->saved_data["options"] = bfly_option_changes();
    Tensor out = layer_fw(twiddle, t2, input, bias, increasing_stride, out_size, wants_grad ? &snapshots : nullptr);
    if (wants_grad) {
      ctx->saved_data["increasing_stride"] = increasing_stride;
      ctx->saved_data["bias"] = bias.has_value() && bias->defined() && bias->requires_grad();
      ctx->save_for_backward({twiddle, t2, input, snapshots});
    }
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_output) {
    auto saved = ctx->get_saved_variables();
    auto r = layer_bw(saved[0], saved[1], saved[2], grad_output[0], ctx->saved_data["increasing_stride"].toBool(),
                      ctx->saved_data["bias"].toBool(), ctx->saved_data["options"].toInt() == bfly_option_changes() ? saved[3] : Tensor());
    return {r.twiddle, r.twiddle2, r.input, r.bias, Tensor(), Tensor(), Tensor()};
  }
};

Tensor butterfly_layer(const Tensor& twiddle, const c10::optional<Tensor>& twiddle2, const Tensor& input,
                       const c10::optional<Tensor>& bias, bool increasing_stride, int64_t out_size) {
  auto needs = [](const c10::optional<Tensor>& t) { return t.has_value() && t->defined() && t->requires_grad(); };
  const bool wants_grad = at::GradMode::is_enabled() && (twiddle.requires_grad() || input.requires_grad() || needs(twiddle2) || needs(bias));
  if (!wants_grad && !has_tangent(twiddle) && !has_tangent(input) && !has_tangent(twiddle2) && !has_tangent(bias))
    return layer_fw(twiddle, twiddle2.has_value() ? *twiddle2 : Tensor(), input, bias, increasing_stride, out_size, nullptr);
  return ButterflyLayer::apply(twiddle, twiddle2, input, bias, increasing_stride, out_size, wants_grad);
}

// The float32 layer on (batch, in_size) rows as stateless operators and as a differentiable one.
void check_linear(const Tensor& twiddle, const Tensor& input) {
  BFLY_CHECK_DIM(input, 2);
  TORCH_CHECK(input.scalar_type() == at::kFloat && twiddle.scalar_type() == at::kFloat, "butterfly_linear: float32 only");
}
Tensor butterfly_linear_fw(const Tensor& twiddle, const Tensor& input, const c10::optional<Tensor>& bias,
                           bool increasing_stride, int64_t out_size) {
  check_linear(twiddle, input);
  return layer_fw(twiddle, Tensor(), input, bias, increasing_stride, out_size, nullptr);
}
// (d_twiddle, d_input (batch, in_size), d_bias (out_size) or an undefined tensor)
std::tuple<Tensor, Tensor, Tensor> butterfly_linear_bw(const Tensor& twiddle, const Tensor& input, const Tensor& grad,
                                                        bool increasing_stride, bool need_bias) {
  check_linear(twiddle, input);
  BFLY_CHECK_DIM(grad, 2);
  auto r = layer_bw(twiddle, Tensor(), input, grad, increasing_stride, need_bias, Tensor());
  return std::make_tuple(r.twiddle, r.input, r.bias);
}
Tensor butterfly_linear(const Tensor& twiddle, const Tensor& input, const c10::optional<Tensor>& bias, bool increasing_stride,
                        int64_t out_size) {
  check_linear(twiddle, input);
  return butterfly_layer(twiddle, c10::nullopt, input, bias, increasing_stride, out_size);
}

// ---------------------------------------------------------------- base-4

struct Base4Shape {
  int64_t batch, nstacks, input_size, nblocks, log_n, n;
};

Base4Shape base4_shape(const Tensor& twiddle4, const Tensor& twiddle2, const Tensor& input, const char* what) {
  BFLY_CHECK_CUDA(twiddle4); BFLY_CHECK_CUDA(twiddle2); BFLY_CHECK_CUDA(input);
  BFLY_CHECK_SAME_DEVICE(twiddle4, input); BFLY_CHECK_SAME_DEVICE(twiddle2, input);
  BFLY_CHECK_DIM(twiddle4, 6); BFLY_CHECK_DIM(twiddle2, 6); BFLY_CHECK_DIM(input, 3);
  Base4Shape s;
  s.batch = input.size(0); s.nstacks = input.size(1); s.input_size = input.size(2);
  s.nblocks = twiddle4.size(1);
  s.log_n = twiddle4.size(2) * 2 + twiddle2.size(2);
  TORCH_CHECK(s.log_n >= 1 && s.log_n <= 24 && twiddle2.size(2) <= 1, what, ": n must be a power of 2");
  s.n = (int64_t)1 << s.log_n;
  if (s.log_n / 2 > 0)
    TORCH_CHECK(twiddle4.sizes() == torch::IntArrayRef({s.nstacks, s.nblocks, s.log_n / 2, s.n / 4, 4, 4}),
                "twiddle4 must have shape (nstacks, nblocks, log_n / 2, n / 4, 4, 4)");
  if (s.log_n % 2 == 1)
    TORCH_CHECK(twiddle2.sizes() == torch::IntArrayRef({s.nstacks, s.nblocks, 1, s.n / 2, 2, 2}),
                "twiddle2 must have shape (nstacks, nblocks, 1, n / 2, 2, 2)");
  TORCH_CHECK((input.scalar_type() == at::kFloat || input.scalar_type() == at::kComplexFloat) &&
                  twiddle4.scalar_type() == input.scalar_type() && twiddle2.scalar_type() == input.scalar_type(),
              what, " not implemented for '", toString(input.scalar_type()), "' (float32 and complex64 only, one dtype)");
  return s;
}

Tensor butterfly_multiply_base4_fw(const Tensor& twiddle4, const Tensor& twiddle2, const Tensor& input,
                                   bool increasing_stride, c10::optional<int64_t> output_size) {
  const Base4Shape s = base4_shape(twiddle4, twiddle2, input, "butterfly_multiply_base4_fw");
  const int64_t out_size = output_size.has_value() ? output_size.value() : s.n;
  TORCH_CHECK(out_size <= s.n && out_size >= 0, "butterfly_multiply_base4_fw: output_size must be <= n");
  c10::cuda::CUDAGuard guard(input.device());
  const Tensor t4 = dense_twiddle(twiddle4), t2 = dense_twiddle(twiddle2);
  const Tensor x = rows_view(input);
  Tensor output = torch::empty({s.batch, s.nstacks, s.n}, input.options());
  auto stream = at::cuda::getCurrentCUDAStream();
  int rc;
  if (input.scalar_type() == at::kFloat) {
    rc = bfly4_fw_f32(t4.numel() ? t4.data_ptr<float>() : nullptr, t2.numel() ? t2.data_ptr<float>() : nullptr,
                      x.data_ptr<float>(), x.stride(0), x.stride(1), output.data_ptr<float>(), (int)s.batch,
                      (int)s.nstacks, (int)s.log_n, (int)s.nblocks, (int)s.input_size, (int)out_size,
                      increasing_stride, stream.stream());
  } else {
    rc = bfly4_fw_c64(t4.numel() ? t4.data_ptr() : nullptr, t2.numel() ? t2.data_ptr() : nullptr, x.data_ptr(),
                      x.stride(0), x.stride(1), output.data_ptr(), (int)s.batch, (int)s.nstacks, (int)s.log_n,
                      (int)s.nblocks, (int)s.input_size, (int)out_size, increasing_stride, stream.stream());
  }
  check_status(rc, "butterfly_multiply_base4_fw");
  return out_size < s.n ? output.slice(2, 0, out_size) : output;
}

std::tuple<Tensor, Tensor, Tensor> butterfly_multiply_base4_bw(const Tensor& twiddle4, const Tensor& twiddle2,
                                                               const Tensor& input, const Tensor& grad,
                                                               bool increasing_stride) {
  const Base4Shape s = base4_shape(twiddle4, twiddle2, input, "butterfly_multiply_base4_bw");
  BFLY_CHECK_CUDA(grad); BFLY_CHECK_SAME_DEVICE(input, grad); BFLY_CHECK_DIM(grad, 3);
  const int64_t out_size = grad.size(2);
  TORCH_CHECK(grad.sizes() == torch::IntArrayRef({s.batch, s.nstacks, out_size}) && out_size <= s.n,
              "grad must have shape (batch_size, nstacks, output_size) with output_size <= n");
  TORCH_CHECK(grad.scalar_type() == input.scalar_type(), "grad must have the dtype of input");
  c10::cuda::CUDAGuard guard(input.device());
  const Tensor t4 = dense_twiddle(twiddle4), t2 = dense_twiddle(twiddle2);
  const Tensor x = rows_view(input), g = rows_view(grad);
  Tensor d4 = torch::empty_like(t4), d2 = torch::empty_like(t2);
  Tensor d_input = torch::empty({s.batch, s.nstacks, std::max(s.input_size, s.n)}, input.options());
  const bool real = input.scalar_type() == at::kFloat;
  const int64_t ws_bytes = bfly4_bw_workspace_bytes(real ? BFLY_F32 : BFLY_C64, (int)s.batch, (int)s.nstacks, (int)s.log_n,
                                                    (int)s.nblocks);
  TORCH_CHECK(ws_bytes >= 0, "butterfly_multiply_base4_bw failed: ", bfly_strerror((int)ws_bytes));
  Tensor ws = torch::empty({ws_bytes}, input.options().dtype(at::kByte));
  auto stream = at::cuda::getCurrentCUDAStream();
  int rc;
  if (real) {
    rc = bfly4_bw_f32(t4.numel() ? t4.data_ptr<float>() : nullptr, t2.numel() ? t2.data_ptr<float>() : nullptr,
                      x.data_ptr<float>(), x.stride(0), x.stride(1), g.data_ptr<float>(), g.stride(0), g.stride(1),
                      d4.numel() ? d4.data_ptr<float>() : nullptr, d2.numel() ? d2.data_ptr<float>() : nullptr,
                      d_input.data_ptr<float>(), (int)s.batch, (int)s.nstacks, (int)s.log_n, (int)s.nblocks,
                      (int)s.input_size, (int)out_size, increasing_stride, ws_bytes ? ws.data_ptr() : nullptr,
                      (size_t)ws_bytes, stream.stream());
  } else {
    rc = bfly4_bw_c64(t4.numel() ? t4.data_ptr() : nullptr, t2.numel() ? t2.data_ptr() : nullptr, x.data_ptr(),
                      x.stride(0), x.stride(1), g.data_ptr(), g.stride(0), g.stride(1),
                      d4.numel() ? d4.data_ptr() : nullptr, d2.numel() ? d2.data_ptr() : nullptr, d_input.data_ptr(),
                      (int)s.batch, (int)s.nstacks, (int)s.log_n, (int)s.nblocks, (int)s.input_size, (int)out_size,
                      increasing_stride, ws_bytes ? ws.data_ptr() : nullptr, (size_t)ws_bytes, stream.stream());
  }
  check_status(rc, "butterfly_multiply_base4_bw");
  if (s.input_size < s.n) d_input = d_input.slice(2, 0, s.input_size);
  return std::make_tuple(d4, d2, d_input);
}

class ButterflyMultiplyBase4 : public torch::autograd::Function<ButterflyMultiplyBase4> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor twiddle4, Tensor twiddle2, Tensor input, bool increasing_stride,
                        c10::optional<int64_t> output_size) {
    ctx->saved_data["increasing_stride"] = increasing_stride;
    ctx->save_for_backward({twiddle4, twiddle2, input});
    return butterfly_multiply_base4_fw(twiddle4, twiddle2, input, increasing_stride, output_size);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_output) {
    auto saved = ctx->get_saved_variables();
    auto r = butterfly_multiply_base4_bw(saved[0], saved[1], saved[2], grad_output[0],
                                         ctx->saved_data["increasing_stride"].toBool());
    return {std::get<0>(r), std::get<1>(r), std::get<2>(r), Tensor(), Tensor()};
  }
};

Tensor butterfly_multiply_base4(const Tensor& twiddle4, const Tensor& twiddle2, const Tensor& input,
                                bool increasing_stride, c10::optional<int64_t> output_size) {
  return ButterflyMultiplyBase4::apply(twiddle4, twiddle2, input, increasing_stride, output_size);
}

// ---------------------------------------------------------------- forward with glue operators
//
// One launch for  [Real2Complex] [gather] butterfly [diagonal] [gather] [real part]  -- the modules
// that surround a Butterfly in the reference's exact transforms (torch_butterfly/special.py,
// permutation.py:65-75, complex_utils.py:100-142, diagonal.py:11-38).  Returns None
// when the rows do not fit a tile (the caller then runs the operators one by one).
c10::optional<Tensor> butterfly_multiply_glue_fw(const Tensor& twiddle, const Tensor& input, bool increasing_stride,
                                  const c10::optional<Tensor>& in_perm, const c10::optional<Tensor>& out_diag,
                                  const c10::optional<Tensor>& out_perm, bool out_real) {
  BFLY_CHECK_CUDA(twiddle); BFLY_CHECK_CUDA(input); BFLY_CHECK_SAME_DEVICE(twiddle, input);
  BFLY_CHECK_DIM(twiddle, 6); BFLY_CHECK_DIM(input, 3);
  const int64_t batch = input.size(0), nstacks = input.size(1), input_size = input.size(2);
  const int64_t nblocks = twiddle.size(1), log_n = twiddle.size(2);
  TORCH_CHECK(log_n >= 1 && log_n <= 24, "butterfly_multiply_glue_fw: n must be a power of 2 (2 <= n <= 2^24)");
  const int64_t n = (int64_t)1 << log_n;
  TORCH_CHECK(twiddle.sizes() == torch::IntArrayRef({nstacks, nblocks, log_n, n / 2, 2, 2}),
              "twiddle must have shape (nstacks, nblocks, log_n, n / 2, 2, 2)");
  TORCH_CHECK(input_size <= n, "butterfly_multiply_glue_fw: input_size must be <= n");
  // (inside the autograd node of glue.py forward mode is off, and the node refuses tangents itself)
  TORCH_CHECK(!c10::AutogradState::get_tls_state().get_fw_grad_mode() || !(has_tangent(twiddle) || has_tangent(input) || has_tangent(out_diag)),
              "butterfly_multiply_glue_fw: forward-mode differentiation is not implemented");
  const bool cplx = twiddle.scalar_type() == at::kComplexFloat;
  TORCH_CHECK(cplx || twiddle.scalar_type() == at::kFloat, "butterfly_multiply_glue_fw: float32 or complex64 twiddle expected");
  const bool x_real = cplx && input.scalar_type() == at::kFloat;
  TORCH_CHECK(x_real || input.scalar_type() == twiddle.scalar_type(), "input must have the dtype of twiddle (or float32 for a complex twiddle)");
  TORCH_CHECK(!out_real || cplx, "out_real needs a complex twiddle");
  auto index_vec = [&](const c10::optional<Tensor>& t, const char* name) -> Tensor {
    if (!t.has_value() || !t->defined()) return Tensor();
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kInt && t->dim() == 1 && t->size(0) == n, name,
                " must be an int32 CUDA vector of n entries");
    return t->contiguous();
  };
  c10::cuda::CUDAGuard guard(input.device());
  const Tensor ip = index_vec(in_perm, "in_perm"), op = index_vec(out_perm, "out_perm");
  Tensor od;
  if (out_diag.has_value() && out_diag->defined()) {
    TORCH_CHECK(out_diag->is_cuda() && out_diag->scalar_type() == twiddle.scalar_type() && out_diag->dim() == 1 &&
                    out_diag->size(0) == n, "out_diag must be a CUDA vector of n entries with the dtype of twiddle");
    od = out_diag->resolve_conj().contiguous();
  }
  TORCH_CHECK(!ip.defined() || input_size == n, "in_perm needs input_size == n");
  const Tensor tw = dense_twiddle(twiddle);
  const Tensor x = rows_view(input);
  Tensor output = torch::empty({batch, nstacks, n}, input.options().dtype(out_real ? at::kFloat : twiddle.scalar_type()));
  auto stream = at::cuda::getCurrentCUDAStream();
  int rc;
  if (cplx) {
    rc = bfly_fw_glue_c64(tw.data_ptr(), x.data_ptr(), x_real, x.stride(0), x.stride(1), output.data_ptr(), out_real,
                          ip.defined() ? ip.data_ptr<int32_t>() : nullptr, od.defined() ? od.data_ptr() : nullptr,
                          op.defined() ? op.data_ptr<int32_t>() : nullptr, (int)batch, (int)nstacks, (int)log_n, (int)nblocks,
                          (int)input_size, (int)n, increasing_stride, stream.stream());
  } else {
    rc = bfly_fw_glue_f32(tw.data_ptr<float>(), x.data_ptr<float>(), x.stride(0), x.stride(1), output.data_ptr<float>(),
                          ip.defined() ? ip.data_ptr<int32_t>() : nullptr, od.defined() ? od.data_ptr<float>() : nullptr,
                          op.defined() ? op.data_ptr<int32_t>() : nullptr, (int)batch, (int)nstacks, (int)log_n, (int)nblocks,
                          (int)input_size, (int)n, increasing_stride, stream.stream());
  }
  if (rc == BFLY_E_UNSUPPORTED) return c10::nullopt;
  check_status(rc, "butterfly_multiply_glue_fw");
  return output;
}

// ---------------------------------------------------------------- unitary twiddle synthesis
//
// (..., 4) float32 angles -> (..., 2, 2) complex64 blocks and back, one kernel each, in place of
// the cos / sin / stack chain of the reference's ButterflyUnitary.forward
// (torch_butterfly/butterfly.py:271-280) and autograd's backward of that chain.
Tensor unitary_twiddle_fw(const Tensor& angles) {
  BFLY_CHECK_CUDA(angles);
  TORCH_CHECK(angles.scalar_type() == at::kFloat && angles.dim() >= 1 && angles.size(-1) == 4,
              "unitary_twiddle: angles must be float32 with last dimension 4 (phi, alpha, psi, chi)");
  c10::cuda::CUDAGuard guard(angles.device());
  const Tensor a = angles.contiguous();
  auto shape = a.sizes().vec();
  shape.back() = 2;
  shape.push_back(2);
  Tensor tw = torch::empty(shape, a.options().dtype(at::kComplexFloat));
  check_status(bfly_unitary_twiddle_fw(a.data_ptr<float>(), tw.data_ptr(), a.numel() / 4, at::cuda::getCurrentCUDAStream().stream()),
               "unitary_twiddle");
  return tw;
}

Tensor unitary_twiddle_bw(const Tensor& angles, const Tensor& grad) {
  BFLY_CHECK_CUDA(angles); BFLY_CHECK_CUDA(grad); BFLY_CHECK_SAME_DEVICE(angles, grad);
  TORCH_CHECK(angles.scalar_type() == at::kFloat && grad.scalar_type() == at::kComplexFloat &&
                  grad.numel() == angles.numel() && angles.dim() >= 1 && angles.size(-1) == 4,
              "unitary_twiddle_bw: angles (..., 4) float32 and grad (..., 2, 2) complex64 expected");
  c10::cuda::CUDAGuard guard(angles.device());
  const Tensor a = angles.contiguous(), g = grad.resolve_conj().contiguous();
  Tensor d = torch::empty_like(a);
  check_status(bfly_unitary_twiddle_bw(a.data_ptr<float>(), g.data_ptr(), d.data_ptr<float>(), a.numel() / 4,
                                       at::cuda::getCurrentCUDAStream().stream()),
               "unitary_twiddle_bw");
  return d;
}

class UnitaryTwiddle : public torch::autograd::Function<UnitaryTwiddle> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor angles) {
    ctx->save_for_backward({angles});
    return unitary_twiddle_fw(angles);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_output) {
    return {unitary_twiddle_bw(ctx->get_saved_variables()[0], grad_output[0])};
  }
};

Tensor unitary_twiddle(const Tensor& angles) { return UnitaryTwiddle::apply(angles); }

// ---------------------------------------------------------------- 2-D maps
//
// Twiddle of the butterfly that applies twiddle1 (size n1) along the low bits and twiddle2 (size n2) along the high bits
// of a flat index of n2 * n1 positions (butterfly_b200/combine.py), and the sums of its gradient onto the two: one
// broadcast copy and one reduction per map and block.
struct KroneckerPart { Tensor view; int64_t dim; };  // a map's factors inside the result; the dimension they repeat along
KroneckerPart kronecker_part(const Tensor& tw, int64_t block, bool first_map, bool inc, int64_t l1, int64_t l2, int64_t h1, int64_t h2) {
  const bool up = inc != (block % 2 == 1);
  const int64_t S = tw.size(0), off = first_map ? (up ? 0 : l2) : (up ? l1 : 0), len = first_map ? l1 : l2;
  Tensor part = tw.select(1, block).narrow(1, off, len);
  // map 1 pairs positions inside a row: pair index = row * n1 / 2 + own; map 2 pairs rows: own * n1 + column
  return first_map ? KroneckerPart{part.view({S, len, 2 * h2, h1, 2, 2}), 2} : KroneckerPart{part.view({S, len, h2, 2 * h1, 2, 2}), 3};
}
class KroneckerTwiddle : public torch::autograd::Function<KroneckerTwiddle> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor t1, Tensor t2, bool inc) {
    const int64_t S = t1.size(0), nb = t1.size(1), l1 = t1.size(2), h1 = t1.size(3), l2 = t2.size(2), h2 = t2.size(3);
    ctx->saved_data["inc"] = inc;
    ctx->saved_data["sizes"] = std::vector<int64_t>{l1, h1, l2, h2};
    Tensor out = torch::empty({S, nb, l1 + l2, 2 * h1 * h2, 2, 2}, t1.options());
    for (int64_t j = 0; j < nb; ++j)
      for (int m = 0; m < 2; ++m) {
        KroneckerPart k = kronecker_part(out, j, m == 0, inc, l1, l2, h1, h2);
        k.view.copy_((m == 0 ? t1 : t2).select(1, j).unsqueeze(k.dim));
      }
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_output) {
    const auto z = ctx->saved_data["sizes"].toIntVector();
    const bool inc = ctx->saved_data["inc"].toBool();
    const Tensor g = grad_output[0].contiguous();
    const int64_t nb = g.size(1);
    variable_list out = {Tensor(), Tensor(), Tensor()};
    for (int m = 0; m < 2; ++m) {
      std::vector<Tensor> blocks;
      for (int64_t j = 0; j < nb; ++j) {
        const KroneckerPart k = kronecker_part(g, j, m == 0, inc, z[0], z[2], z[1], z[3]);
        blocks.push_back(k.view.sum(k.dim));
      }
      out[m] = nb == 1 ? blocks[0].unsqueeze(1) : torch::stack(blocks, 1);
    }
    return out;
  }
};
// The same from views and one cat per block, which every transform has rules for; the node above has none for forward
// mode and functorch.
Tensor kronecker_composed(const Tensor& t1, const Tensor& t2, bool inc) {
  const int64_t S = t1.size(0), nb = t1.size(1), l1 = t1.size(2), h1 = t1.size(3), l2 = t2.size(2), h2 = t2.size(3);
  const Tensor a = t1.unsqueeze(3).expand({S, nb, l1, 2 * h2, h1, 2, 2}).reshape({S, nb, l1, 2 * h2 * h1, 2, 2});
  const Tensor b = t2.unsqueeze(4).expand({S, nb, l2, h2, 2 * h1, 2, 2}).reshape({S, nb, l2, h2 * 2 * h1, 2, 2});
  std::vector<Tensor> blocks;
  for (int64_t j = 0; j < nb; ++j) {
    const bool up = inc != (j % 2 == 1);
    blocks.push_back(torch::cat({(up ? a : b).select(1, j), (up ? b : a).select(1, j)}, 1));
  }
  return torch::stack(blocks, 1);
}
Tensor kronecker_twiddle(const Tensor& twiddle1, const Tensor& twiddle2, bool increasing_stride) {
  BFLY_CHECK_DIM(twiddle1, 6); BFLY_CHECK_DIM(twiddle2, 6); BFLY_CHECK_SAME_DEVICE(twiddle1, twiddle2);
  TORCH_CHECK(twiddle1.size(0) == twiddle2.size(0) && twiddle1.size(1) == twiddle2.size(1) && twiddle1.scalar_type() == twiddle2.scalar_type(),
              "kronecker_twiddle: the two maps must have the same stacks, blocks and dtype");
  if (has_tangent(twiddle1) || has_tangent(twiddle2) || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
    return kronecker_composed(twiddle1, twiddle2, increasing_stride);
  return KroneckerTwiddle::apply(twiddle1, twiddle2, increasing_stride);
}

// The reference's import-time check (torch_butterfly/__init__.py:13-31) compares this
// with torch.version.cuda, so report the CUDA runtime torch itself runs on.
int64_t cuda_version() { return at::detail::getCUDAHooks().versionCUDART(); }

int64_t launch_count() { return bfly_launch_count(); }

}  // namespace

TORCH_LIBRARY(torch_butterfly, m) {
  m.def("butterfly_multiply_fw(Tensor twiddle, Tensor input, bool increasing_stride, int? output_size=None) -> Tensor",
        butterfly_multiply_fw);
  m.def("butterfly_multiply_bw(Tensor twiddle, Tensor input, Tensor grad, bool increasing_stride) -> (Tensor, Tensor)",
        butterfly_multiply_bw);
  m.def("butterfly_multiply(Tensor twiddle, Tensor input, bool increasing_stride, int? output_size=None) -> Tensor",
        butterfly_multiply);
  m.def("butterfly_linear_fw(Tensor twiddle, Tensor input, Tensor? bias, bool increasing_stride, int out_size) -> Tensor",
        butterfly_linear_fw);
  m.def("butterfly_linear_bw(Tensor twiddle, Tensor input, Tensor grad, bool increasing_stride, bool need_bias) -> (Tensor, Tensor, Tensor)",
        butterfly_linear_bw);
  m.def("butterfly_linear(Tensor twiddle, Tensor input, Tensor? bias, bool increasing_stride, int out_size) -> Tensor",
        butterfly_linear);
  m.def("butterfly_layer(Tensor twiddle, Tensor? twiddle2, Tensor input, Tensor? bias, bool increasing_stride, int out_size) -> Tensor",
        butterfly_layer);
  m.def("butterfly_multiply_glue_fw(Tensor twiddle, Tensor input, bool increasing_stride, Tensor? in_perm, Tensor? out_diag, Tensor? out_perm, bool out_real) -> Tensor?",
        butterfly_multiply_glue_fw);
  m.def("unitary_twiddle_fw(Tensor angles) -> Tensor", unitary_twiddle_fw);
  m.def("unitary_twiddle_bw(Tensor angles, Tensor grad) -> Tensor", unitary_twiddle_bw);
  m.def("unitary_twiddle(Tensor angles) -> Tensor", unitary_twiddle);
  m.def("kronecker_twiddle(Tensor twiddle1, Tensor twiddle2, bool increasing_stride) -> Tensor", kronecker_twiddle);
  m.def("butterfly_multiply_base4_fw(Tensor twiddle4, Tensor twiddle2, Tensor input, bool increasing_stride, int? output_size=None) -> Tensor",
        butterfly_multiply_base4_fw);
  m.def("butterfly_multiply_base4_bw(Tensor twiddle4, Tensor twiddle2, Tensor input, Tensor grad, bool increasing_stride) -> (Tensor, Tensor, Tensor)",
        butterfly_multiply_base4_bw);
  m.def("butterfly_multiply_base4(Tensor twiddle4, Tensor twiddle2, Tensor input, bool increasing_stride, int? output_size=None) -> Tensor",
        butterfly_multiply_base4);
#ifndef BFLY_SEPARATE_VERSION_LIB
  m.def("cuda_version() -> int", cuda_version);
#endif
  m.def("b200_launch_count() -> int", launch_count);
}

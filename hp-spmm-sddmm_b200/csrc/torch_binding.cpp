// PyTorch operators of the aggregation layer, in C++: registration, autograd formula, stream and memory handling.
//
// A training step on a small graph is three or four launches of a few microseconds each; with the operators and the
// autograd formula in Python the host took 160 us to issue them.  Arithmetic stays in libhpspmm.so, which this file
// calls through the C ABI; PyTorch supplies memory, streams and the autograd tape.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <memory>
#include <mutex>
#include <unordered_map>

#include "hpspmm.h"

namespace {

using at::Tensor;

struct Entry {
  // Held while a call uses the handles and the fields below: the interpreter lock is not held then, and threads may meet
  // on one layer (the autograd engine's and the caller's at least).
  std::mutex use;
  hpspmm_ctx* ctx;
  hpspmm_layer* layer;   // null once the layer is closed
  int64_t M, N, nnz;
  // the weight tensor whose values the layer's transpose holds (kept alive: the layer borrows the device array)
  Tensor vals;
  int64_t vals_version;   // of `vals` when the transpose was filled; -1: unknown, fill it again
  bool in_graph = false;  // a captured graph fills the transpose: a replay does so without the host knowing
};

std::mutex g_mutex;   // guards the registry
std::unordered_map<int64_t, std::shared_ptr<Entry>> g_layers;

std::shared_ptr<Entry> entry_of(int64_t id) {
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_layers.find(id);
  TORCH_CHECK(it != g_layers.end(), "hpspmm: unknown or closed layer id ", id);
  return it->second;
}

void check_open(const Entry& e, int64_t id) { TORCH_CHECK(e.layer, "hpspmm: unknown or closed layer id ", id); }

void check(const Entry& e, int status, const char* what) {
  TORCH_CHECK(status == HPSPMM_OK, what, " failed with status ", status, ": ", hpspmm_last_error(e.ctx));
}

Tensor require_cuda_f32(const Tensor& t, int64_t rows, const char* what) {
  TORCH_CHECK(t.is_cuda(), "hpspmm: ", what, " must be a CUDA tensor (there is no CPU path)");
  TORCH_CHECK(t.scalar_type() == at::kFloat && t.dim() == 2 && t.size(0) == rows, "hpspmm: ", what,
              " must be float32 of shape [", rows, ", K], got ", t.scalar_type(), " ", t.sizes());
  return t.contiguous();
}

Tensor require_weights(const Tensor& t, const Entry& e, const at::Device& device) {
  TORCH_CHECK(t.is_cuda() && t.device() == device && t.scalar_type() == at::kFloat && t.numel() >= e.nnz,
              "hpspmm: vals must be ", e.nnz, " float32 values on ", device, ", got ", t.scalar_type(), " ", t.sizes(), " on ",
              t.device());
  return t.contiguous();
}

// Re-gathers the transpose's values when the weight tensor moved or was written in place.  What was held goes to `old`, to
// be released after the lock.
// A captured call always records the gather: its graph may be replayed after the weights changed in place, or after a call
// with others.  From then on nobody knows what the transpose holds, and every call gathers.
void sync_values(Entry& e, const Tensor& vals, cudaStream_t stream, Tensor& old) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture != cudaStreamCaptureStatusNone) e.in_graph = true;
  const int64_t version = vals.is_inference() || e.in_graph ? -1 : (int64_t)vals._version();
  if (version >= 0 && e.vals.defined() && vals.const_data_ptr() == e.vals.const_data_ptr() && version == e.vals_version)
    return;
  e.vals_version = -1;   // until the update has succeeded
  check(e, hpspmm_layer_update_values(e.ctx, e.layer, vals.const_data_ptr<float>(), stream), "hpspmm_layer_update_values");
  old = std::move(e.vals);
  e.vals = vals.detach();
  e.vals_version = version;
}

Tensor forward(const Tensor& H, const Tensor& vals, int64_t id) {
  auto e = entry_of(id);
  const Tensor h = require_cuda_f32(H, e->N, "H"), v = require_weights(vals, *e, H.device());
  const c10::cuda::CUDAGuard guard(h.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  Tensor C = at::empty({e->M, h.size(1)}, h.options());
  std::lock_guard<std::mutex> lock(e->use);
  check_open(*e, id);
  check(*e, hpspmm_layer_forward_values(e->ctx, e->layer, h.size(1), v.const_data_ptr<float>(), h.const_data_ptr<float>(),
                                        C.mutable_data_ptr<float>(), stream), "hpspmm_layer_forward");
  return C;
}

Tensor backward_features(const Tensor& grad, const Tensor& vals, int64_t id) {
  auto e = entry_of(id);
  const Tensor dC = require_cuda_f32(grad, e->M, "dC"), v = require_weights(vals, *e, grad.device());
  const c10::cuda::CUDAGuard guard(dC.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  Tensor dH = at::empty({e->N, dC.size(1)}, dC.options());
  Tensor old;
  std::lock_guard<std::mutex> lock(e->use);
  check_open(*e, id);
  sync_values(*e, v, stream, old);
  check(*e, hpspmm_layer_backward_features(e->ctx, e->layer, dC.size(1), dC.const_data_ptr<float>(),
                                           dH.mutable_data_ptr<float>(), stream), "hpspmm_layer_backward_features");
  return dH;
}

Tensor backward_weights(const Tensor& grad, const Tensor& H, int64_t id) {
  auto e = entry_of(id);
  const Tensor dC = require_cuda_f32(grad, e->M, "dC");
  const Tensor h = require_cuda_f32(H, e->N, "H");
  TORCH_CHECK(h.size(1) == dC.size(1), "hpspmm: dC and H differ in width");
  const c10::cuda::CUDAGuard guard(dC.device());
  Tensor dA = at::empty({e->nnz}, dC.options());
  std::lock_guard<std::mutex> lock(e->use);
  check_open(*e, id);
  check(*e, hpspmm_layer_backward_weights(e->ctx, e->layer, dC.size(1), dC.const_data_ptr<float>(),
                                          h.const_data_ptr<float>(), dA.mutable_data_ptr<float>(),
                                          c10::cuda::getCurrentCUDAStream().stream()), "hpspmm_layer_backward_weights");
  return dA;
}

// Both gradients: one pass over the transpose where the library has a kernel for the call, else the product and the SDDMM,
// into the same tensors.
std::tuple<Tensor, Tensor> backward(const Tensor& grad, const Tensor& H, const Tensor& vals, int64_t id) {
  auto e = entry_of(id);
  const Tensor dC = require_cuda_f32(grad, e->M, "dC"), h = require_cuda_f32(H, e->N, "H");
  const Tensor v = require_weights(vals, *e, grad.device());
  TORCH_CHECK(h.size(1) == dC.size(1) && h.device() == dC.device(), "hpspmm: dC and H differ in width or device");
  const c10::cuda::CUDAGuard guard(dC.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  Tensor dH = at::empty({e->N, dC.size(1)}, dC.options()), dA = at::empty({e->nnz}, dC.options());
  const int64_t K = dC.size(1);
  const float *dc = dC.const_data_ptr<float>(), *hp = h.const_data_ptr<float>();
  float *dh = dH.mutable_data_ptr<float>(), *da = dA.mutable_data_ptr<float>();
  Tensor old;
  std::lock_guard<std::mutex> lock(e->use);
  check_open(*e, id);
  const int st = hpspmm_layer_backward(e->ctx, e->layer, K, v.const_data_ptr<float>(), dc, hp, dh, da, stream);
  if (st != HPSPMM_ERR_UNSUPPORTED) {
    check(*e, st, "hpspmm_layer_backward");
    return {dH, dA};
  }
  sync_values(*e, v, stream, old);
  check(*e, hpspmm_layer_backward_features(e->ctx, e->layer, K, dc, dh, stream), "hpspmm_layer_backward_features");
  check(*e, hpspmm_layer_backward_weights(e->ctx, e->layer, K, dc, hp, da, stream), "hpspmm_layer_backward_weights");
  return {dH, dA};
}

// the registered operators, for calls that go through the dispatcher (tracing, fake tensors)
using Op = Tensor(const Tensor&, const Tensor&, int64_t);
c10::TypedOperatorHandle<Op> find_op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Op>();
}
const c10::TypedOperatorHandle<Op>& op_forward() {
  static const auto op = find_op("hpspmm::layer_forward");
  return op;
}
const c10::TypedOperatorHandle<Op>& op_features() {
  static const auto op = find_op("hpspmm::layer_backward_features");
  return op;
}
const c10::TypedOperatorHandle<Op>& op_weights() {
  static const auto op = find_op("hpspmm::layer_backward_weights");
  return op;
}

using OpBoth = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, int64_t);
const c10::TypedOperatorHandle<OpBoth>& op_both() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("hpspmm::layer_backward", "").typed<OpBoth>();
  return op;
}

struct LayerFunction : public torch::autograd::Function<LayerFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& H, const Tensor& vals, int64_t id) {
    ctx->saved_data["id"] = id;
    ctx->save_for_backward({H, vals});
    at::AutoDispatchBelowADInplaceOrView below;
    return op_forward().call(H, vals, id);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const int64_t id = ctx->saved_data["id"].toInt();
    Tensor dH, dvals;
    if (grads[0].defined()) {
      const bool features = ctx->needs_input_grad(0), weights = ctx->needs_input_grad(1);
      if (features && weights)
        std::tie(dH, dvals) = op_both().call(grads[0], saved[0], saved[1], id);
      else if (features)
        dH = op_features().call(grads[0], saved[1], id);
      else if (weights)
        dvals = op_weights().call(grads[0], saved[0], id);
    }
    return {dH, dvals, Tensor()};
  }
};

Tensor forward_autograd(const Tensor& H, const Tensor& vals, int64_t id) { return LayerFunction::apply(H, vals, id); }

// The two gradients have no derivative of their own.  Without a formula on the autograd key PyTorch would only warn and
// leave their terms out of a second derivative, so differentiating them is an error.
template <const c10::TypedOperatorHandle<Op>& (*OP)()>
struct NoDerivative : public torch::autograd::Function<NoDerivative<OP>> {
  static Tensor forward(torch::autograd::AutogradContext*, const Tensor& a, const Tensor& b, int64_t id) {
    at::AutoDispatchBelowADInplaceOrView below;
    return OP().call(a, b, id);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext*, torch::autograd::variable_list) {
    TORCH_CHECK(false, "hpspmm: no derivative of ", OP().schema().name(), " is implemented (a second derivative of the layer)");
  }
};
template <const c10::TypedOperatorHandle<Op>& (*OP)()>
Tensor gradient_autograd(const Tensor& a, const Tensor& b, int64_t id) {
  if (at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad())) return NoDerivative<OP>::apply(a, b, id);
  at::AutoDispatchBelowADInplaceOrView below;
  return OP().call(a, b, id);
}

struct NoDerivativeOfBoth : public torch::autograd::Function<NoDerivativeOfBoth> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext*, const Tensor& dC, const Tensor& H,
                                                const Tensor& vals, int64_t id) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto out = op_both().call(dC, H, vals, id);
    return {std::get<0>(out), std::get<1>(out)};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext*, torch::autograd::variable_list) {
    TORCH_CHECK(false, "hpspmm: no derivative of ", op_both().schema().name(),
                " is implemented (a second derivative of the layer)");
  }
};
std::tuple<Tensor, Tensor> both_autograd(const Tensor& dC, const Tensor& H, const Tensor& vals, int64_t id) {
  if (at::GradMode::is_enabled() && (dC.requires_grad() || H.requires_grad() || vals.requires_grad())) {
    auto out = NoDerivativeOfBoth::apply(dC, H, vals, id);
    return {out[0], out[1]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return op_both().call(dC, H, vals, id);
}

TORCH_LIBRARY(hpspmm, m) {
  m.def("layer_forward(Tensor H, Tensor vals, int layer_id) -> Tensor");
  m.def("layer_backward_features(Tensor dC, Tensor vals, int layer_id) -> Tensor");
  m.def("layer_backward_weights(Tensor dC, Tensor H, int layer_id) -> Tensor");
  m.def("layer_backward(Tensor dC, Tensor H, Tensor vals, int layer_id) -> (Tensor, Tensor)");
}
// a CPU tensor reaches the same functions, which refuse it by name
#define HPSPMM_IMPL(KEY)                                  \
  TORCH_LIBRARY_IMPL(hpspmm, KEY, m) {                    \
    m.impl("layer_forward", forward);                     \
    m.impl("layer_backward_features", backward_features); \
    m.impl("layer_backward_weights", backward_weights);   \
    m.impl("layer_backward", backward);                   \
  }
HPSPMM_IMPL(CUDA)
HPSPMM_IMPL(CPU)
TORCH_LIBRARY_IMPL(hpspmm, Autograd, m) {
  m.impl("layer_forward", forward_autograd);
  m.impl("layer_backward_features", gradient_autograd<op_features>);
  m.impl("layer_backward_weights", gradient_autograd<op_weights>);
  m.impl("layer_backward", both_autograd);
}

void register_layer(int64_t id, int64_t ctx, int64_t layer, int64_t M, int64_t N, int64_t nnz, const Tensor& vals) {
  auto e = std::make_shared<Entry>();
  e->ctx = reinterpret_cast<hpspmm_ctx*>(ctx);
  e->layer = reinterpret_cast<hpspmm_layer*>(layer);
  e->M = M, e->N = N, e->nnz = nnz;
  e->vals = vals.detach();
  e->vals_version = vals.is_inference() ? -1 : (int64_t)vals._version();
  std::lock_guard<std::mutex> lock(g_mutex);
  g_layers[id] = e;
}

// The caller destroys the handles next: calls in flight end first, later ones find the layer closed.
void forget_layer(int64_t id) {
  std::shared_ptr<Entry> e;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    auto it = g_layers.find(id);
    if (it == g_layers.end()) return;
    e = std::move(it->second);
    g_layers.erase(it);
  }
  std::lock_guard<std::mutex> lock(e->use);
  e->layer = nullptr;
}

}  // namespace

PYBIND11_MODULE(_hpspmm_torch, m) {
  m.def("register_layer", &register_layer);
  m.def("forget_layer", &forget_layer, py::call_guard<py::gil_scoped_release>());
  m.def("layer_forward", [](const Tensor& H, const Tensor& vals, int64_t id) { return op_forward().call(H, vals, id); },
        py::call_guard<py::gil_scoped_release>());
}

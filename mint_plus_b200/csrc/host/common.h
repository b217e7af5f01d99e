// Host side of the operators in C++: tensors in, launches of libmintb out, without the interpreter in between.
//
// A step of a small model is a few hundred launches of a few microseconds each, and from Python every one of them cost the host
// 20 to 35 us (argument conversion, tensor wrappers, a Python autograd function): the 8M training step ran 11.1 ms for 2.3 ms of
// kernels, one pair through the FP8 650M model 13.9 ms for 3.5 ms.  Here a launch costs the driver call, its tensor maps and the
// allocator; the backward pass runs on autograd's thread without the interpreter lock.
#pragma once

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <optional>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../../include/mintb.h"

namespace mintb_host {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// A CUDA failure reported by the library (the Python side maps it to MintbError).
struct MintbFailure : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline void check(int rc, const char* what) {
  if (rc == MINTB_OK) return;
  const std::string msg = std::string(what) + ": " + mintb_last_error();
  if (rc == MINTB_EINVAL || rc == MINTB_EWORKSPACE) TORCH_CHECK_VALUE(false, msg);
  if (rc == MINTB_EUNSUPPORTED) TORCH_CHECK_NOT_IMPLEMENTED(false, msg);
  throw MintbFailure(msg);
}

Tensor dev_status(int device);   // the device's status word (int32 [1]), created on first use

// Everything a launch needs to know about where it runs; makes the tensor's device current for its lifetime.
struct Env {
  explicit Env(const Tensor& t) : guard(t.device()), stream(at::cuda::getCurrentCUDAStream(t.device().index()).stream()), status(status_ptr(t.device().index())), opts(t.options()) {}
  c10::cuda::CUDAGuard guard;
  void* stream;
  int* status;
  at::TensorOptions opts;   // options of the tensor: device, layout (dtype overridden per allocation)

  // (straight to the allocator: a training step of the 8M model makes 330 of these, and the dispatcher is a third of what one costs)
  Tensor empty(at::IntArrayRef sizes, at::ScalarType dt) const { return at::detail::empty_cuda(sizes, dt, opts.device(), std::nullopt); }
  Tensor bytes(size_t n) const { return n ? empty({int64_t(n)}, at::kByte) : Tensor(); }

 private:
  static int* status_ptr(int device);
};

inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
inline Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

inline int dt_code(at::ScalarType t, const char* what) {
  switch (t) {
    case at::kFloat: return MINTB_F32;
    case at::kBFloat16: return MINTB_BF16;
    case at::kFloat8_e4m3fn: return MINTB_E4M3;
    case at::kFloat8_e5m2: return MINTB_E5M2;
    default: TORCH_CHECK_TYPE(false, what, " has an unsupported dtype");
  }
}
inline int param_dt(const Tensor& t, const char* what) {
  if (!t.defined()) return MINTB_F32;
  TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16, what, " must be float32 or bfloat16");
  return dt_code(t.scalar_type(), what);
}
// rows [first, first + n) of a tensor, as a view
inline Tensor rows_of(const Tensor& t, int64_t first, int64_t n) {
  c10::SmallVector<int64_t, 4> sizes(t.sizes());
  sizes[0] = n;
  return t.as_strided(sizes, t.strides(), t.storage_offset() + first * t.stride(0));
}
inline Tensor as_dtype(const Tensor& t, at::ScalarType dt) { return !t.defined() || t.scalar_type() == dt ? t : t.to(dt); }

// ---- launches (no autograd) ---------------------------------------------------------------------------------------------------

struct AttnInputs {   // (B,H,T,D) projections and what goes with them
  Tensor q[6];        // q, k, v of the self pathway, then of the cross pathway
  Tensor meta, cos, sin;
  double scale;
  unsigned flags;
  Tensor ids, pad;    // forward: `meta` is still to be filled from these chain ids and this key padding (bytes)
};
struct AttnResult {
  Tensor out, lse;
  Tensor q8;          // `out` in e4m3, where asked for
  Tensor ws;          // workspace holding the rotated copies the backward pass starts from, where asked for
};
AttnResult attn_fwd(const AttnInputs& a, bool for_backward, double q8_scale = 0.0);   // q8_scale > 0 (bf16): with the e4m3 copy

struct Product {      // y = act(alpha x w^T + bias) and its variants
  Tensor x, w, bias;
  double alpha = 1.0;
  bool gelu = false, save_preact = false;
  double out_e4m3 = 0.0;         // scale of an e4m3 result, 0: bf16
};
std::pair<Tensor, Tensor> linear_fwd(const Product& p);     // (y, pre-activation)
// res_a resid + res_b (alpha x w^T + bias), and with quant > 0 its e4m3 copy saturate(. / quant); round_first: the projection is rounded
// to bf16 before the sum
std::pair<Tensor, Tensor> linear_res_fwd(const Product& p, const Tensor& resid, double res_a, double res_b, double quant, bool round_first = false);
// fp32: act(x w^T + bias) (+ resid) of (rows, K) rows
Tensor linear_f32(const Tensor& x, const Tensor& w, const OptTensor& bias, bool gelu, const OptTensor& resid);
// fp32: the q, k, v projections of (T,B,E) activations, head-major: `w` and `bias` hold the weights in order, each [E][E] or [3E][E]
std::vector<Tensor> heads_f32(const Tensor& x, const std::vector<Tensor>& w, const std::vector<OptTensor>& bias, int64_t H);
Tensor quantize(const Tensor& x, double scale);
// alpha (dz w + dz2 w2) + beta resid
Tensor dgrad(const Tensor& dz, const Tensor& w, double alpha, const Tensor& dz2 = {}, const Tensor& w2 = {}, const Tensor& resid = {}, double beta = 0.0);
Tensor wgrad(const Tensor& dz, const Tensor& x, double alpha, at::ScalarType out);
// Weight gradients of several projections over the same tokens, formed by one launch: dw = alpha dz^T x, db (where wanted) the column
// sums of dz, in bf16.
struct WeightGrad {
  Tensor dz, x, dw, db;
  double alpha = 1.0;
  bool want_db = false;
};
void wgrad_group(std::vector<WeightGrad>& items);
// (dz, db): dz = dy gelu'(z) (dy itself without z) in bf16, db its column sums in the given type (none: not wanted)
std::pair<Tensor, Tensor> gelu_colsum(const Tensor& dy, const Tensor& z, std::optional<at::ScalarType> db_dt);
// (dz in e5m2, db)
std::pair<Tensor, Tensor> gelu_colsum_f8(const Tensor& dy, const Tensor& z, std::optional<at::ScalarType> db_dt, double scale);
// Bytes that the caching allocator holds on the device without using them.
int64_t cached_free_bytes(int device);
// The capture that the current stream of the tensor's device is in, 0 if none.
uint64_t capture_id(const Tensor& t);

struct NormOut {
  Tensor s, y, stats, q8;
};
NormOut add_layernorm_fwd(const Tensor& x, const Tensor& r, double a, double b, const Tensor& gamma, const Tensor& beta, double eps, bool need_s, double quant);
struct NormGrad {
  Tensor dx, dr, dgamma, dbeta;   // parameter gradients in the type of gamma
};
NormGrad add_layernorm_bwd(const Tensor& dy, const Tensor& ds, const Tensor& x, const Tensor& r, double a, double b, const Tensor& gamma, const Tensor& stats,
                           bool want_params, bool ds_apart = false);   // ds_apart: ds is added to the rounded dx

// The operators have no forward-mode derivative: a tangent on an input is an error and not dropped.
inline void no_tangent(const Tensor& t) {
  TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), "mint_plus_b200 operators have no forward-mode derivative");
}

// Which inputs of a call want gradients, as a node of the autograd graph; nullptr when none does.
template <typename N>
std::shared_ptr<N> make_node(const std::vector<Tensor>& inputs) {
  for (const Tensor& t : inputs) no_tangent(t);
  if (!at::GradMode::is_enabled()) return nullptr;
  bool any = false;
  for (const Tensor& t : inputs) any = any || (t.defined() && t.requires_grad());
  if (!any) return nullptr;
  auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
  torch::autograd::edge_list edges;
  edges.reserve(inputs.size());
  for (const Tensor& t : inputs) edges.push_back(t.defined() ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge());
  node->set_next_edges(std::move(edges));
  return node;
}

}  // namespace mintb_host

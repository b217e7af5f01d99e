#pragma once

#include "ops.h"

namespace mintb_host {

// The static scale of an e5m2 gradient cast, kept on the Python side; 0 until a first backward pass has measured it.
struct ScaleHolder {
  virtual ~ScaleHolder() = default;
  virtual double current() = 0;
  virtual double fix(double amax) = 0;   // the scale for gradients of that size, from now on
};

// One projection's operand: the bf16 weight itself, or its e4m3 copy with the scales of an 8-bit product.
struct Operand {
  Tensor w;
  double w_scale = 1.0, x_scale = 1.0, out_scale = 1.0;
  double grad_scale = 0.0;   // of the e5m2 cast of its output gradient; 0: ask the holder
  std::shared_ptr<ScaleHolder> holder;
  double alpha() const { return w_scale * x_scale * out_scale; }
};

// What a batch brings with it.
struct Batch {
  int64_t T, B;
  Tensor meta, cos, sin;
  Tensor rows32, rows64, inv32;   // packed tokens: (t, b) row of each token, and its inverse; undefined: the padded grid
};

// A two-pathway transformer layer laid out for calling: its parameters and the operands formed from them.  The Python layer builds
// one and keeps it while state() finds the parameters what they were.
struct LayerPlan {
  bool mu = false;      // x = keep x + add attn(x); x = LN(keep x + add ffn(x)); else x += attn(LN(x)); x += ffn(LN(x))
  bool fp8 = false, sqrt_softmax = false;
  int64_t H = 0, D = 0;
  double scale = 1.0, keep = 1.0, add = 1.0, eps1 = 0.0, eps2 = 0.0;
  // parameters: self q/k/v weights (one fused or three), their biases, the cross pathway's, then out, fc1, fc2 (weight, bias) and the
  // norms (gamma, beta): the first one on Pre-LN layers only.  An absent bias is undefined.  They are the module's own tensors, so a
  // product that reads one directly follows whatever is written to it or put in its place.
  std::vector<Tensor> params;
  int64_t n_self = 1, n_cross = 1;
  Operand qkv_self, qkv_cross, out, fc1, fc2;   // qkv operands [3E][E], rows [Q; K; V]
  // frozen projections with adapters: params ends with A and B of self q, k, v, cross q, k, v and out; the operands are formed per call
  int64_t lora_r = 0;
  double lora_scaling = 1.0;
  bool joint = false;                           // both pathways' projections are one product: on
  Tensor qkv6, bias6;                           // this operand, a copy that is kept while its sources stand
  Tensor bias_self, bias_cross;                 // [3E] biases of separate products

  // Forms what is copied from the parameters (not the e4m3 weights, which Python hands in) and notes what it was copied from.
  void form();
  // kCurrent; kWritten: a parameter behind a kept copy has been written or replaced since, and form() takes it in; kOther: the plan was
  // laid out for something else (another type, or e4m3 copies of weights that have changed).
  enum State { kCurrent, kWritten, kOther };
  int state() const;
  LayerPlan refreshed() const;   // (a plan of its own: calls under way keep theirs)
  std::tuple<Tensor, OptTensor> forward(const Tensor& x, const OptTensor& xq, const Batch& batch, double next_quant) const;

 private:
  struct Stamp {
    at::ScalarType dtype;
    bool copied;        // a kept copy depends on it
    const void* data;
    uint32_t version;
  };
  std::vector<Stamp> stamps;   // one for each parameter
  std::tuple<Tensor, OptTensor> run(const Tensor& x, const OptTensor& xq, const Batch& batch, double next_quant) const;
};

}  // namespace mintb_host

#pragma once

#include <array>

#include "common.h"

namespace mintb_host {

// The attention's gradients as rows of the fused projections' output: row t * B + b of a [rows][3E] matrix, or row token_row[t * B + b]
// (negative: none) when only some tokens have one; with tables the self pathway's dq, dk are un-rotated on the way.
struct RowMajor {
  int64_t rows;
  Tensor token_row, cos, sin;
};
// Gradients of the six inputs; with `rm` the two matrices in [0] and [1].
std::array<Tensor, 6> attn_bwd(const AttnInputs& a, const Tensor& out, const Tensor& lse, const Tensor& d_out, const Tensor& saved_ws, const RowMajor* rm);

// Metadata blob of a (B,T) batch from chain ids and (optionally) padded keys.
Tensor mask_meta(const Tensor& chain_ids, const OptTensor& key_pad);
// (with chain_ids the metadata is formed here and `meta` is not read)
Tensor attention(std::array<Tensor, 6> qkv, const Tensor& meta, const OptTensor& cos, const OptTensor& sin, double scale, int64_t flags, const OptTensor& chain_ids = {},
                 const OptTensor& key_pad = {});
Tensor combine(const Tensor& il, const Tensor& el, const Tensor& mask_u8, const Tensor& iv, const Tensor& ev);
Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& bias, bool gelu);
std::tuple<OptTensor, OptTensor, OptTensor> add_layernorm(const Tensor& x, const OptTensor& r, double a, double b, const OptTensor& gamma, const OptTensor& beta,
                                                          double eps, bool need_s, double quant);
Tensor embed(const Tensor& tokens, const Tensor& weight, int64_t pad, int64_t mask, bool dropout, double ratio);
std::tuple<Tensor, Tensor> mlm_corrupt(const Tensor& tokens, const Tensor& u_target, const Tensor& u_kind, const Tensor& residue, int64_t cls, int64_t eos, int64_t pad,
                                       int64_t mask);   // (corrupted tokens, targets)
Tensor masked_ce(const Tensor& logits, const Tensor& targets, const Tensor& target_mask);

}  // namespace mintb_host

// Differentiable operators: each is one node of the autograd graph over the launches of launch.cpp.
#include "ops.h"

#include <tuple>

namespace mintb_host {

using torch::autograd::set_history;

static Tensor rows_of(const Tensor& x) { return x.reshape({-1, x.size(-1)}).contiguous(); }

// ---- attention ----------------------------------------------------------------------------------------------------------------
std::array<Tensor, 6> attn_bwd(const AttnInputs& a, const Tensor& out, const Tensor& lse, const Tensor& d_out, const Tensor& saved_ws, const RowMajor* rm) {
  const Tensor& q = a.q[0];
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2), D = q.size(3), E = H * D;
  const int dt = dt_code(q.scalar_type(), "q");
  Env e(q);
  unsigned flags = a.flags;
  std::array<Tensor, 6> grads;
  void* g[6];
  Tensor cos = a.cos, sin = a.sin;
  if (rm != nullptr) {   // straight into the [rows][3E] matrices [dQ | dK | dV] of the projections, un-rotated
    for (int p = 0; p < 2; ++p) {
      grads[p] = e.empty({rm->rows, 3 * E}, q.scalar_type());
      for (int k = 0; k < 3; ++k) g[3 * p + k] = static_cast<char*>(grads[p].data_ptr()) + size_t(k) * E * 2;
    }
    cos = rm->cos;
    sin = rm->sin;
    if (cos.defined()) flags |= MINTB_FLAG_ROPE | MINTB_FLAG_QK_PREROTATED;
    flags |= MINTB_FLAG_GRAD_ROWMAJOR;
  } else {
    for (int k = 0; k < 6; ++k) {
      grads[k] = e.empty({B, H, T, D}, q.scalar_type());
      g[k] = grads[k].data_ptr();
    }
  }
  size_t bytes = mintb_attn_bwd_workspace_bytes(B, H, T, D, dt, flags);
  Tensor ws = saved_ws;
  if (ws.defined()) {
    bytes = ws.numel();
    flags |= MINTB_FLAG_ROT_SAVED;
  } else {
    ws = e.bytes(bytes);
  }
  check(mintb_attn_bwd_rows(ptr(a.q[0]), ptr(a.q[1]), ptr(a.q[2]), ptr(a.q[3]), ptr(a.q[4]), ptr(a.q[5]), ptr(a.meta), fptr(cos), fptr(sin), ptr(out),
                            fptr(lse), ptr(d_out), g[0], g[1], g[2], g[3], g[4], g[5], ptr(ws), bytes, B, H, T, D, dt, flags, float(a.scale), e.stream,
                            e.status, rm != nullptr && rm->token_row.defined() ? rm->token_row.data_ptr<int32_t>() : nullptr),
        "mintb_attn_bwd");
  return grads;
}

struct AttentionNode : public torch::autograd::Node {
  SavedVariable q[6], out, lse, ws;
  Tensor meta, cos, sin;
  double scale = 1.0;
  unsigned flags = 0;
  variable_list apply(variable_list&& grads) override {
    variable_list r(6);
    if (!grads[0].defined()) return r;
    at::NoGradGuard no_grad;
    AttnInputs a;
    for (int k = 0; k < 6; ++k) a.q[k] = q[k].unpack();
    a.meta = meta; a.cos = cos; a.sin = sin; a.scale = scale; a.flags = flags;
    auto g = attn_bwd(a, out.unpack(shared_from_this()), lse.unpack(), grads[0].contiguous(), ws.unpack(), nullptr);
    for (int k = 0; k < 6; ++k) r[k] = g[k];
    return r;
  }
  void release_variables() override {
    for (auto& s : q) s.reset_data();
    out.reset_data(); lse.reset_data(); ws.reset_data();
  }
  std::string name() const override { return "MultimerAttentionBackward"; }
};

// Chain ids and key padding as the metadata kernels read them.
static std::pair<Tensor, Tensor> mask_inputs(const Tensor& chain_ids, const OptTensor& key_pad) {
  at::NoGradGuard no_grad;
  TORCH_CHECK(chain_ids.is_cuda(), "mint_plus_b200 operators run on CUDA tensors only (no CPU fallback)");
  TORCH_CHECK_VALUE(chain_ids.dim() == 2, "chain_ids must be (B, T)");
  Tensor ids = chain_ids.scalar_type() == at::kLong || chain_ids.scalar_type() == at::kInt ? chain_ids.contiguous() : chain_ids.to(at::kInt).contiguous();
  Tensor pad = opt(key_pad);
  if (pad.defined()) {
    TORCH_CHECK(pad.is_cuda(), "mint_plus_b200 operators run on CUDA tensors only (no CPU fallback)");
    TORCH_CHECK_VALUE(pad.sizes() == chain_ids.sizes(), "key_padding_mask must be (B, T) = ", chain_ids.sizes(), ", got ", pad.sizes());
    pad = pad.contiguous();
    pad = pad.scalar_type() == at::kBool ? pad.view(at::kByte) : pad.to(at::kByte);
  }
  return {ids, pad};
}

Tensor mask_meta(const Tensor& chain_ids, const OptTensor& key_pad) {
  at::NoGradGuard no_grad;
  auto [ids, pad] = mask_inputs(chain_ids, key_pad);
  const int64_t B = ids.size(0), T = ids.size(1);
  Env e(ids);
  Tensor buf = e.bytes(mintb_mask_meta_bytes(B, T));
  if (ids.scalar_type() == at::kLong)
    check(mintb_mask_meta_from_chain_ids64(ids.data_ptr<int64_t>(), static_cast<uint8_t*>(ptr(pad)), ptr(buf), B, T, e.stream), "mask_meta_from_chain_ids");
  else
    check(mintb_mask_meta_from_chain_ids(ids.data_ptr<int32_t>(), static_cast<uint8_t*>(ptr(pad)), ptr(buf), B, T, e.stream), "mask_meta_from_chain_ids");
  return buf;
}

Tensor attention(std::array<Tensor, 6> qkv, const Tensor& meta, const OptTensor& cos, const OptTensor& sin, double scale, int64_t flags, const OptTensor& chain_ids,
                 const OptTensor& key_pad) {
  for (const Tensor& t : qkv) TORCH_CHECK(t.is_cuda(), "mint_plus_b200 operators run on CUDA tensors only (no CPU fallback)");
  for (const Tensor& t : qkv)
    TORCH_CHECK_VALUE(t.dim() == 4 && t.sizes() == qkv[0].sizes(), "q/k/v of both pathways must share one (B, H, T, D) shape");
  for (const Tensor& t : qkv)
    TORCH_CHECK_TYPE(t.scalar_type() == qkv[0].scalar_type() && (t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16),
                     "q/k/v must all be float32 or all be bfloat16");
  AttnInputs a;
  std::vector<Tensor> in(6);
  for (int k = 0; k < 6; ++k) a.q[k] = in[k] = qkv[k].contiguous();
  a.meta = meta; a.cos = opt(cos); a.sin = opt(sin); a.scale = scale; a.flags = unsigned(flags);
  if (chain_ids.has_value()) {   // (of the batch of q, on its device: the caller has looked)
    std::tie(a.ids, a.pad) = mask_inputs(*chain_ids, key_pad);
    a.meta = Env(a.ids).bytes(mintb_mask_meta_bytes(int(a.ids.size(0)), int(a.ids.size(1))));
  }
  auto node = make_node<AttentionNode>(in);
  AttnResult r = attn_fwd(a, node != nullptr);
  if (node) {
    set_history(r.out, node);
    for (int k = 0; k < 6; ++k) node->q[k] = SavedVariable(a.q[k], false);
    node->out = SavedVariable(r.out, true);
    node->lse = SavedVariable(r.lse, false); node->ws = SavedVariable(r.ws, false);
    node->meta = a.meta; node->cos = a.cos; node->sin = a.sin;
    node->scale = scale; node->flags = a.flags;
  }
  return r.out;
}

// ---- combine from logits ------------------------------------------------------------------------------------------------------
struct CombineNode : public torch::autograd::Node {
  SavedVariable il, el, iv, ev;
  Tensor mask;
  variable_list apply(variable_list&& grads) override {
    variable_list r(4);
    if (!grads[0].defined()) return r;
    at::NoGradGuard no_grad;
    const Tensor l0 = il.unpack(), l1 = el.unpack(), v0 = iv.unpack(), v1 = ev.unpack(), g = grads[0].contiguous();
    const int64_t B = v0.size(0), H = v0.size(1), T = v0.size(2), D = v0.size(3);
    Env e(v0);
    r[0] = e.empty(l0.sizes(), l0.scalar_type());
    r[1] = e.empty(l0.sizes(), l0.scalar_type());
    r[2] = e.empty(v0.sizes(), v0.scalar_type());
    r[3] = e.empty(v0.sizes(), v0.scalar_type());
    const size_t bytes = mintb_combine_bwd_workspace_bytes(B, H, T);
    Tensor ws = e.bytes(bytes);
    check(mintb_combine_bwd(ptr(l0), ptr(l1), mask.data_ptr<uint8_t>(), ptr(v0), ptr(v1), ptr(g), ptr(r[0]), ptr(r[1]), ptr(r[2]), ptr(r[3]), ptr(ws), bytes, B, H,
                            T, D, dt_code(v0.scalar_type(), "values"), e.stream),
          "mintb_combine_bwd");
    return r;
  }
  void release_variables() override {
    for (SavedVariable* s : {&il, &el, &iv, &ev}) s->reset_data();
    mask = Tensor();
  }
  std::string name() const override { return "MultimerCombineBackward"; }
};

Tensor combine(const Tensor& il_, const Tensor& el_, const Tensor& mask_u8, const Tensor& iv_, const Tensor& ev_) {
  const Tensor il = il_.contiguous(), el = el_.contiguous(), iv = iv_.contiguous(), ev = ev_.contiguous();
  const int64_t B = iv.size(0), H = iv.size(1), T = iv.size(2), D = iv.size(3);
  Env e(iv);
  Tensor out = e.empty(iv.sizes(), iv.scalar_type());
  check(mintb_combine_fwd(ptr(il), ptr(el), mask_u8.data_ptr<uint8_t>(), ptr(iv), ptr(ev), ptr(out), B, H, T, D, dt_code(iv.scalar_type(), "values"), e.stream),
        "mintb_combine_fwd");
  if (auto node = make_node<CombineNode>({il, el, iv, ev})) {
    set_history(out, node);
    node->il = SavedVariable(il, false); node->el = SavedVariable(el, false);
    node->iv = SavedVariable(iv, false); node->ev = SavedVariable(ev, false);
    node->mask = mask_u8;
  }
  return out;
}

// ---- plain projection ---------------------------------------------------------------------------------------------------------
// The products take rows of 16-byte multiples: a weight with other numbers of rows (the vocabulary) gets zero rows appended.
static Tensor pad_rows(const Tensor& t, int64_t n) {
  Env e(t);
  auto shape = t.sizes().vec();
  shape[0] = n;
  Tensor out = e.empty(shape, t.scalar_type());
  const size_t have = t.nbytes(), all = out.nbytes();
  cudaStream_t s = static_cast<cudaStream_t>(e.stream);
  C10_CUDA_CHECK(cudaMemcpyAsync(out.data_ptr(), t.data_ptr(), have, cudaMemcpyDeviceToDevice, s));
  C10_CUDA_CHECK(cudaMemsetAsync(static_cast<char*>(out.data_ptr()) + have, 0, all - have, s));
  return out;
}

struct LinearNode : public torch::autograd::Node {
  SavedVariable x, w, z;
  Tensor padded;      // the weight with its zero rows, where it has any
  int64_t n = 0;      // its rows without them
  std::vector<int64_t> x_shape;
  at::ScalarType w_dt = at::kBFloat16, b_dt = at::kBFloat16;
  bool has_bias = false;
  variable_list apply(variable_list&& grads) override {
    variable_list r(3);
    if (!grads[0].defined()) return r;
    at::NoGradGuard no_grad;
    const Tensor x2 = rows_of(x.unpack());
    Tensor dy;
    if (padded.defined()) {
      auto shape = x_shape;
      shape.back() = padded.size(0);
      dy = at::zeros(shape, x2.options());
      dy.narrow(-1, 0, n).copy_(grads[0]);
      dy = dy.view({x2.size(0), -1});
    } else {
      dy = grads[0].reshape({x2.size(0), -1}).contiguous();
    }
    const bool want_db = has_bias && task_should_compute_output(2);
    const Tensor wt = as_dtype(w.unpack(), at::kBFloat16).contiguous();
    auto [dz, db] = gelu_colsum(dy, z.unpack(), want_db ? std::optional<at::ScalarType>(b_dt) : std::nullopt);
    if (task_should_compute_output(0)) r[0] = dgrad(dz, padded.defined() ? padded : wt, 1.0).view(x_shape);
    if (task_should_compute_output(1)) r[1] = as_dtype(wgrad(dz, x2, 1.0, w_dt == at::kFloat ? at::kFloat : at::kBFloat16), w_dt);
    if (want_db) r[2] = db;
    if (padded.defined())
      for (int k = 1; k < 3; ++k)
        if (r[k].defined()) r[k] = rows_of(r[k], 0, n);
    return r;
  }
  void release_variables() override {
    x.reset_data(); w.reset_data(); z.reset_data(); padded.reset();
  }
  std::string name() const override { return "LinearBackward"; }
};

Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& bias_, bool gelu) {
  const Tensor bias = opt(bias_);
  auto node = make_node<LinearNode>({x, w, bias});
  Tensor y, z;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    Product p;
    p.x = rows_of(x);
    p.w = as_dtype(w, at::kBFloat16).contiguous();
    p.bias = bias.defined() ? bias.contiguous() : bias;
    p.gelu = gelu;
    p.save_preact = node != nullptr;
    const int64_t n = w.size(0), np = (n + 7) / 8 * 8;
    if (np != n) {
      p.w = pad_rows(p.w, np);
      if (bias.defined()) p.bias = pad_rows(p.bias, np);
      if (node) { node->padded = p.w; node->n = n; }
    }
    Tensor out;
    std::tie(out, z) = linear_fwd(p);
    auto shape = x.sizes().vec();
    shape.back() = np;
    y = out.view(shape);
    if (np != n) y = y.narrow(-1, 0, n);
  }
  if (node) {
    set_history(y, node);
    node->x = SavedVariable(x, false);
    node->w = SavedVariable(w, false);
    node->z = SavedVariable(z, false);
    node->has_bias = bias.defined();
    node->x_shape = x.sizes().vec();
    node->w_dt = w.scalar_type();
    if (bias.defined()) node->b_dt = bias.scalar_type();
  }
  return y;
}

// ---- residual sum and LayerNorm -----------------------------------------------------------------------------------------------
struct AddNormNode : public torch::autograd::Node {
  SavedVariable x, r, gamma, stats;
  std::vector<int64_t> shape;
  double a = 1.0, b = 0.0;
  bool has_r = false, norm = false, has_beta = false, has_s = false;
  at::ScalarType p_dt = at::kBFloat16;
  variable_list apply(variable_list&& grads) override {
    variable_list res(4);
    Tensor ds = has_s ? grads[0] : Tensor(), dy = norm ? grads[has_s ? 1 : 0] : Tensor();
    if (!ds.defined() && !dy.defined()) return res;
    at::NoGradGuard no_grad;
    const Tensor x2 = rows_of(x.unpack()), r2 = has_r ? rows_of(r.unpack()) : Tensor();
    if (ds.defined()) ds = rows_of(ds);
    if (dy.defined()) dy = rows_of(dy);
    else if (norm) dy = at::zeros_like(x2);
    const bool want = norm && (task_should_compute_output(2) || task_should_compute_output(3));   // frozen parameters: no sums at all
    NormGrad g = add_layernorm_bwd(dy, ds, x2, r2, a, b, norm ? gamma.unpack() : Tensor(), stats.unpack(), want);
    res[0] = g.dx.view(shape);
    if (has_r) res[1] = g.dr.view(shape);
    if (want) {
      res[2] = as_dtype(g.dgamma, p_dt);
      if (has_beta) res[3] = as_dtype(g.dbeta, p_dt);
    }
    return res;
  }
  void release_variables() override {
    x.reset_data(); r.reset_data(); gamma.reset_data(); stats.reset_data();
  }
  std::string name() const override { return "AddLayerNormBackward"; }
};

std::tuple<OptTensor, OptTensor, OptTensor> add_layernorm(const Tensor& x, const OptTensor& r_, double a, double b, const OptTensor& gamma_, const OptTensor& beta_,
                                                          double eps, bool need_s, double quant) {
  const Tensor r = opt(r_), gamma = opt(gamma_), beta = opt(beta_);
  auto node = make_node<AddNormNode>({x, r, gamma, beta});
  NormOut o;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    o = add_layernorm_fwd(rows_of(x), r.defined() ? rows_of(r) : r, a, b, gamma, beta, eps, need_s, quant);
    if (o.s.defined()) o.s = o.s.view(x.sizes());
    if (o.y.defined()) o.y = o.y.view(x.sizes());
  }
  if (node) {
    if (o.s.defined()) set_history(o.s, node);
    if (o.y.defined()) set_history(o.y, node);
    node->x = SavedVariable(x, false);
    if (r.defined()) node->r = SavedVariable(r, false);
    if (gamma.defined()) {
      node->gamma = SavedVariable(gamma, false);
      node->p_dt = gamma.scalar_type();
    }
    node->stats = SavedVariable(o.stats, false);
    node->shape = x.sizes().vec();
    node->a = a; node->b = b;
    node->has_r = r.defined(); node->norm = gamma.defined(); node->has_beta = beta.defined(); node->has_s = o.s.defined();
  }
  auto some = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
  return {some(o.s), some(o.y), some(o.q8)};
}

// ---- the model's ends ---------------------------------------------------------------------------------------------------------
struct EmbedNode : public torch::autograd::Node {
  Tensor tokens, scales;
  int64_t V = 0, E = 0, pad = 0, mask = 0;
  bool dropout = false;
  at::ScalarType dt = at::kBFloat16;
  variable_list apply(variable_list&& grads) override {
    variable_list r(1);
    if (!grads[0].defined()) return r;
    at::NoGradGuard no_grad;
    Tensor g = grads[0].contiguous();
    if (reinterpret_cast<uintptr_t>(g.data_ptr()) % 16) g = g.clone();   // a view off the kernel's alignment
    Env e(g);
    Tensor dw = e.empty({V, E}, at::kFloat);
    check(mintb_embed_bwd(reinterpret_cast<const long long*>(tokens.data_ptr<int64_t>()), ptr(g), fptr(scales), fptr(dw), tokens.size(0), tokens.size(1), E, V,
                          dt_code(dt, "weight"), pad, mask, dropout, e.stream),
          "mintb_embed_bwd");
    r[0] = as_dtype(dw, dt);
    return r;
  }
  void release_variables() override { tokens = scales = Tensor(); }
  std::string name() const override { return "EmbedTokensBackward"; }
};

Tensor embed(const Tensor& tokens, const Tensor& weight, int64_t pad, int64_t mask, bool dropout, double ratio) {
  Env e(weight);
  const int64_t B = tokens.size(0), T = tokens.size(1), V = weight.size(0), E = weight.size(1);
  auto node = make_node<EmbedNode>({weight});
  Tensor out = e.empty({T, B, E}, weight.scalar_type()), scales = e.empty({B}, at::kFloat);
  Tensor w;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    w = weight.contiguous();
  }
  check(mintb_embed_fwd(reinterpret_cast<const long long*>(tokens.data_ptr<int64_t>()), ptr(w), ptr(out), fptr(scales), B, T, E, V,
                        dt_code(weight.scalar_type(), "weight"), pad, mask, dropout, float(ratio), e.stream),
        "mintb_embed_fwd");
  if (node) {
    set_history(out, node);
    node->tokens = tokens; node->scales = scales; node->V = V; node->E = E; node->pad = pad; node->mask = mask; node->dropout = dropout;
    node->dt = weight.scalar_type();
  }
  return out;
}

struct MaskedCeNode : public torch::autograd::Node {
  SavedVariable logits, lse, sums;
  Tensor targets, mask;
  int64_t N = 0, ld = 0, V = 0;
  variable_list apply(variable_list&& grads) override {
    variable_list r(1);
    if (!grads[0].defined()) return r;
    at::NoGradGuard no_grad;
    const Tensor l = logits.unpack();
    Env e(l);
    Tensor d = e.empty({N, ld}, at::kBFloat16);
    const Tensor g = grads[0].to(at::kFloat).reshape({1}).contiguous();
    check(mintb_masked_ce_bwd(ptr(l), reinterpret_cast<const long long*>(targets.data_ptr<int64_t>()), mask.data_ptr<uint8_t>(), fptr(lse.unpack()), fptr(sums.unpack()), fptr(g), ptr(d),
                              N, ld, V, e.stream),
          "mintb_masked_ce_bwd");
    r[0] = d.as_strided(l.sizes(), l.strides(), 0);
    return r;
  }
  void release_variables() override {
    logits.reset_data(); lse.reset_data(); sums.reset_data();
    targets = mask = Tensor();
  }
  std::string name() const override { return "MaskedCrossEntropyBackward"; }
};

std::tuple<Tensor, Tensor> mlm_corrupt(const Tensor& tokens, const Tensor& u_target, const Tensor& u_kind, const Tensor& residue, int64_t cls, int64_t eos, int64_t pad,
                                       int64_t mask) {
  Env e(tokens);
  Tensor out = e.empty(tokens.sizes(), at::kLong), target = e.empty(tokens.sizes(), at::kBool);
  auto i64 = [](const Tensor& t) { return reinterpret_cast<long long*>(t.data_ptr<int64_t>()); };
  check(mintb_mlm_corrupt(i64(tokens), fptr(u_target), fptr(u_kind), i64(residue), i64(out), reinterpret_cast<unsigned char*>(target.data_ptr<bool>()), tokens.numel(),
                          int(cls), int(eos), int(pad), int(mask), e.stream),
        "mintb_mlm_corrupt");
  return {out, target};
}

Tensor masked_ce(const Tensor& logits_, const Tensor& targets_, const Tensor& target_mask) {
  const int64_t B = logits_.size(0), T = logits_.size(1), V = logits_.size(2);
  Tensor logits = logits_, tg = targets_, mk = target_mask;
  int64_t ld;
  if (logits.stride(0) == T * logits.stride(1)) {          // rows in (B, T) order
    ld = logits.stride(1);
  } else if (logits.stride(1) == B * logits.stride(0)) {   // rows in (T, B) order: a transposed view
    ld = logits.stride(0);
    tg = tg.t();
    mk = mk.t();
  } else {
    logits = logits.contiguous();
    ld = V;
  }
  auto node = make_node<MaskedCeNode>({logits});
  at::AutoDispatchBelowADInplaceOrView below;
  Env e(logits);
  const int64_t N = B * T;
  tg = tg.contiguous();
  mk = mk.contiguous();
  mk = mk.scalar_type() == at::kBool ? mk.view(at::kByte) : mk.to(at::kByte);
  Tensor lse = e.empty({N}, at::kFloat), sums = e.empty({2}, at::kFloat);
  check(mintb_masked_ce_fwd(ptr(logits), reinterpret_cast<const long long*>(tg.data_ptr<int64_t>()), mk.data_ptr<uint8_t>(), fptr(lse), fptr(sums), N, ld, V, e.stream),
        "mintb_masked_ce_fwd");
  Tensor loss = at::div(sums.select(0, 0), sums.select(0, 1));
  if (node) {
    set_history(loss, node);
    node->logits = SavedVariable(logits, false);
    node->lse = SavedVariable(lse, false); node->sums = SavedVariable(sums, false);
    node->targets = tg; node->mask = mk; node->N = N; node->ld = ld; node->V = V;
  }
  return loss;
}

}  // namespace mintb_host

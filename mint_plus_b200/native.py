"""Lays the two-pathway layers out for the C++ host side (csrc/host/layer.cpp): which parameters and operands a layer's forward
and backward pass take, formed once and kept on the layer until one of them changes.

A layer is served here when it is what the builders make: bf16 activations on the GPU, nn.Linear projections with bf16 weights
(with or without LoRA adapters on a frozen base) or Fp8Linear ones throughout, LayerNorms with parameters, the fused attention, a
VanillaFeedForward, and none of the methods that this file stands in for overridden.

The modules' own path (modules_plus.py, mu_scaling.py on the operators of ops.py) serves the rest, and has to stay for it:
* layers with fp32 weights under bf16 activations, RMSNorm, mixed kinds of projections or foreign ones, blocks and attentions of a subclass;
* LoRA with dropout, on fused or on some projections only, of a rank that is no multiple of eight, on trainable bases or above 1870 columns;
* FP8 layers without 8-bit gradients while gradients are on, or whose pathways have different activation scales, and calibration;
* layers while hooks are registered on their block or a wrapped output projection, or module-wide ones;
* MINTB_FUSE_OUT_RESIDUAL=0, the materialised-logits combine, single-pathway layers;
* everything in fp32 with gradients: run_layer_f32 at the end of this file serves plain fp32 Pre-LN layers without them.
"""
from __future__ import annotations

from typing import Optional

import torch
from torch import nn
from torch.nn.modules.module import _has_any_global_hook as _any_global_hook

from . import _lib as L
from . import ops


class _Plan:
    """The native plan of a layer and what it was made from: `slots` are (dict, key, object) that must still hold that object
    (the contents behind the copied operands the native plan watches), `fixed` the layer's own settings; `hooks` are the hook
    dictionaries of the modules that would be called otherwise: while one is filled the layer runs through the modules.  The layer keeps
    its plan and the plan nothing of the layer's own dictionary: a dropped layer dies at once, weights and copies with it."""

    __slots__ = ("native", "slots", "fixed", "hooks", "can_grad", "x_scale", "rot", "block")

    def valid(self, fixed) -> bool:
        if self.fixed != fixed:
            return False
        for d, k, o in self.slots:
            if d.get(k) is not o:
                return False
        state = self.native.state()
        if state == 1 and not torch.cuda.is_current_stream_capturing():     # (a captured call joins its weights itself)
            self.native = self.native.refreshed()
        return state < 2

    # copies of a model lay their layers out themselves
    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return type(None), ()


_ATTN_CHILDREN = ("q_proj", "k_proj", "v_proj", "fused_qkv", "out_proj", "rot_emb")


def _attn_mods(attn):
    fused = attn._modules.get("fused_qkv")
    mods = [fused] if fused is not None else [attn._modules.get(n) for n in ("q_proj", "k_proj", "v_proj")]
    return None if any(m is None for m in mods) else mods


def _own(mp, obj, *names) -> bool:
    """These methods of `obj` are the package's, overridden neither in a subclass nor on the instance nor patched."""
    return all(getattr(getattr(obj, n, None), "__func__", None) in mp.OWN_CODE for n in names)


def _hooks(mod):
    return [mod._forward_hooks, mod._forward_pre_hooks, mod._backward_hooks, mod._backward_pre_hooks]


def _build(layer, mu: bool, fixed) -> Optional[_Plan]:
    from . import modules_plus as mp
    from .lora import LoRALinear
    from .mu_scaling import Fp8Linear, fused_fp8_weight
    sa, ma, ff = layer.self_attn, layer.multimer_attn, layer.feed_forward
    ms, mc = _attn_mods(sa), _attn_mods(ma)
    if ms is None or mc is None or sa._modules.get("out_proj") is None or type(ff) is not mp.VanillaFeedForward:
        return None
    one = [sa.out_proj, ff.fc1, ff.fc2]
    adapters = None
    if all(type(m) is LoRALinear for m in ms + mc + one[:1]):
        adapters = ms + mc + one[:1]
        if len(ms) != 3 or len(mc) != 3 or len({(m.r, m.scaling) for m in adapters}) != 1 or adapters[0].r % 8 or sa.embed_dim % 8 or \
                12 * sa.embed_dim ** 2 > mp._QKV6_MAX_BYTES or any(isinstance(m.dropout, nn.Dropout) or type(m.base) is not nn.Linear for m in adapters):
            return None
        ms, mc, one = [m.base for m in ms], [m.base for m in mc], [one[0].base] + one[1:]
        if any(p.dtype != torch.bfloat16 or not p.is_contiguous() for m in adapters for p in (m.lora_A, m.lora_B)) or \
                any(p.requires_grad for m in ms + mc + one[:1] for p in m.parameters()):
            return None
    linears = ms + mc + one
    fp8 = type(linears[0]) is Fp8Linear
    if any(type(m) is not (Fp8Linear if fp8 else nn.Linear) for m in linears) or (fp8 and any(m._observing for m in linears)):
        return None
    for mods in (ms, mc):
        if len({m.bias is None for m in mods}) != 1 or len({m.weight.dtype for m in mods}) != 1:
            return None
    norms = [layer.final_layer_norm] if mu else [layer.self_attn_layer_norm, layer.final_layer_norm]
    params_dt = (torch.bfloat16, torch.float32)
    if any(type(n) is not nn.LayerNorm or n.weight is None or n.weight.dtype not in params_dt for n in norms):
        return None
    if any(m.weight.dtype not in ((torch.bfloat16,) if not fp8 else params_dt) or not m.weight.is_cuda or not m.weight.is_contiguous()
           or (m.bias is not None and (m.bias.dtype not in params_dt or not m.bias.is_contiguous())) for m in linears):
        return None
    E, H = sa.embed_dim, sa.num_heads
    keep, add, sqrt_softmax = fixed
    bias_s, bias_c = ms[0].bias is not None, mc[0].bias is not None

    p = _Plan()
    p.slots, p.fixed = [], fixed
    for m, names in ((layer, ("self_attn", "multimer_attn", "feed_forward", "final_layer_norm") + (() if mu else ("self_attn_layer_norm",))),
                     (sa, _ATTN_CHILDREN), (ma, _ATTN_CHILDREN), (ff, ("fc1", "fc2"))):
        p.slots += [(m._modules, n, m._modules.get(n)) for n in names]
    for m in linears + norms:
        p.slots += [(m._parameters, "weight", m._parameters.get("weight")), (m._parameters, "bias", m._parameters.get("bias"))]
    p.slots += [(sa.__dict__, k, sa.__dict__.get(k)) for k in ("scaling", "num_heads", "head_dim")] + [(n.__dict__, "eps", n.eps) for n in norms]

    p.block, p.hooks = ff, _hooks(ff)
    if adapters is not None:
        p.hooks += _hooks(adapters[-1])
        p.slots += [(adapters[-1].__dict__, "forward", None)]
    for m in adapters or ():
        p.slots += [(m._modules, n, m._modules.get(n)) for n in ("base", "dropout")] + [(m._parameters, n, m._parameters.get(n)) for n in ("lora_A", "lora_B")]
        p.slots += [(m.__dict__, "scaling", m.__dict__.get("scaling"))]

    # both pathways' projections as one product that reads x once; a larger [6E][E] operand pushes the activation rows out of L2 between
    # column tiles (measured slower)
    joint = adapters is None and mp.FUSE_QKV6 and 6 * E * E * (1 if fp8 else 2) <= mp._QKV6_MAX_BYTES and bias_s == bias_c
    qkv6 = None
    if fp8:
        f8s, f8c = fused_fp8_weight(sa, ms), fused_fp8_weight(ma, mc)
        if f8s[2] != f8c[2]:
            return None          # one cast of the input serves both products
        holders = [f8s[4], one[0].grad_scale, one[1].grad_scale, one[2].grad_scale]
        p.can_grad = all(m.fp8_grads for m in linears)
        op_s = L.host().Operand(f8s[0], f8s[1], f8s[2], f8s[3], holders[0])
        op_c = L.host().Operand(f8c[0], f8c[1], f8c[2], f8c[3])
        wq = [m._quantized_weight() for m in one]
        o, f1, f2 = (L.host().Operand(w, s, m.x_scale, m.out_scale, h) for (w, s), m, h in zip(wq, one, holders[1:]))
        for m in linears:
            p.slots += [(m.__dict__, k, m.__dict__.get(k)) for k in ("_wq", "x_scale", "out_scale", "fp8_grads", "grad_scale", "_observing")]
        p.slots += [(h.__dict__, "scale", h.scale) for h in holders if h is not None]
        p.slots += [(a.__dict__, "_fp8_qkv_grad_scale", a.__dict__.get("_fp8_qkv_grad_scale")) for a in (sa, ma)]
        p.x_scale = f8s[2]
        if joint:
            with ops.normal_tensors():
                qkv6 = torch.cat([f8s[0].view(torch.uint8), f8c[0].view(torch.uint8)]).view(torch.float8_e4m3fn)
    else:
        p.can_grad, p.x_scale = True, 0.0
        if adapters is not None and bias_s != bias_c:
            return None
        op_s = op_c = L.host().Operand(None)
        o, f1, f2 = (L.host().Operand(m.weight) for m in one)
    params = [m.weight for m in ms] + [m.bias for m in ms] + [m.weight for m in mc] + [m.bias for m in mc]
    for m in one + norms:
        params += [m.weight, m.bias]
    if adapters is not None:
        params += [m.lora_A for m in adapters] + [m.lora_B for m in adapters]
    p.native = L.host().LayerPlan(mu=mu, fp8=fp8, sqrt_softmax=sqrt_softmax, H=H, D=sa.head_dim, scale=sa.scaling, keep=keep, add=add,
                                  eps1=norms[0].eps, eps2=norms[-1].eps, params=params, n_self=len(ms), n_cross=len(mc), qkv_self=op_s, qkv_cross=op_c,
                                  out=o, fc1=f1, fc2=f2, joint=joint, qkv6=qkv6, lora_r=adapters[0].r if adapters else 0, lora_scaling=adapters[0].scaling if adapters else 1.0)
    p.rot = sa.rot_emb
    return p


def run_layer(layer, x, chain_mask, padding_mask, chain_ids, pack, *, mu: bool, keep: float, add: float, next_quant=None):
    """The layer's result for x (T,B,E) (or the packed rows of one), or None when the layer is not served here."""
    from . import modules_plus as mp
    if not (x.is_cuda and x.dtype == torch.bfloat16 and layer.use_multimer and layer._use_fused_multi_pathway and mp.FUSE_OUT_RESIDUAL and
            getattr(layer._multimer_attention_superfused, "__func__", None) in mp.OWN_CODE):
        return None
    plan = layer.__dict__.get("_native_plan")
    fixed = (keep, add, bool(layer._use_sqrt_softmax))
    if plan is None or not plan.valid(fixed):
        if layer.self_attn.head_dim not in (16, 32, 64):
            return None
        plan = _build(layer, mu, fixed)
        if not ops.capture_id(x):     # (what a capture forms exists in its replays only)
            layer.__dict__["_native_plan"] = plan
        if plan is None:
            return None
    if ((not plan.can_grad and torch.is_grad_enabled()) or any(plan.hooks) or _any_global_hook() or
            getattr(plan.block.forward, "__func__", None) not in mp.OWN_CODE):
        return None
    T, B = (pack.T, pack.B) if pack is not None else (x.shape[0], x.shape[1])
    meta = mp._cached_ids_meta(chain_ids, padding_mask) if chain_ids is not None and chain_mask is None else ops.cached_mask_meta(chain_mask, padding_mask)
    cos = sin = None
    if plan.rot is not None:
        cos, sin, _ = ops.rope_tables(T, layer.self_attn.head_dim, x.device, plan.rot.inv_freq)
    xq = ops.attached_e4m3(x, plan.x_scale) if mu and plan.x_scale else None
    rows = (pack.rows32, pack.rows64, pack.inv32) if pack is not None else (None, None, None)
    y, q8 = plan.native.forward(x, xq, T, B, meta.buf, cos, sin, *rows, next_quant or 0.0)
    if q8 is not None:
        ops.attach_e4m3(y, q8, next_quant)
    return y


def _plain(mod, kind, dtype=torch.float32) -> bool:
    """`mod` is exactly a `kind` with aligned contiguous parameters of `dtype` and no hooks."""
    return (type(mod) is kind and not any(_hooks(mod)) and "forward" not in mod.__dict__ and
            all(p is None or (p.is_cuda and p.dtype == dtype and p.is_contiguous() and p.data_ptr() % 16 == 0) for p in (mod.weight, mod.bias)))


def run_layer_f32(layer, x, chain_mask, padding_mask, chain_ids):
    """The Pre-LN layer's result for fp32 activations (T,B,E) without gradients, or None when the layer is not served here: every
    projection one launch with bias, GELU and residual sum in its epilogue, and the six of q, k, v together with the head-major
    layout.  (With gradients the projections stay autograd's linears, which keep what their backward pass needs.)"""
    from . import modules_plus as mp
    if (torch.is_grad_enabled() or not (x.is_cuda and x.dtype == torch.float32 and x.is_contiguous() and x.data_ptr() % 16 == 0) or
            not (layer.use_multimer and layer._use_fused_multi_pathway) or layer._use_sqrt_softmax or torch.is_autocast_enabled("cuda")):
        return None
    sa, ma, ff = layer.self_attn, layer.multimer_attn, layer.feed_forward
    if type(ff) is not mp.VanillaFeedForward or sa.head_dim not in (16, 32, 64) or x.numel() == 0:
        return None
    if any(_hooks(ff)) or _any_global_hook():
        return None
    if not (_own(mp, layer, "_multimer_attention_plus", "_multimer_attention_superfused") and _own(mp, ff, "forward") and
            all(_own(mp, a, "project_qkv_4d") and (not hasattr(a, "_project_qkv") or _own(mp, a, "_project_qkv")) for a in (sa, ma))):
        return None
    projections = [m for a in (sa, ma) for m in (_attn_mods(a) or [None])]
    if not (all(m is not None and _plain(m, torch.nn.Linear) for m in (*projections, sa.out_proj, ff.fc1, ff.fc2)) and ff.fc1.out_features % 4 == 0 and
            type(layer.self_attn_layer_norm) is type(layer.final_layer_norm) is torch.nn.LayerNorm):
        return None
    T, B, E = x.shape
    host = L.host()
    meta = mp._cached_ids_meta(chain_ids, padding_mask) if chain_ids is not None and chain_mask is None else ops.cached_mask_meta(chain_mask, padding_mask)
    rope = sa.rot_emb is not None
    heads = host.heads_f32(layer.self_attn_layer_norm(x), [m.weight for m in projections], [m.bias for m in projections], sa.num_heads)
    out = ops.multimer_attention(*heads, meta=meta, rope=rope, inv_freq=sa.rot_emb.inv_freq if rope else None, scale=sa.scaling, out_seq_first=True)
    x = host.linear_f32(out.reshape(T, B, E), sa.out_proj.weight, sa.out_proj.bias, False, x)
    h = host.linear_f32(layer.final_layer_norm(x), ff.fc1.weight, ff.fc1.bias, True, None)
    return host.linear_f32(h, ff.fc2.weight, ff.fc2.bias, False, x)

"""The work that users have this package do, as cases that a timing harness can run: `listed()`, more of the same ranges from
`draw(rng)`, and for each case `prepare`, `run`, `work` and `tolerance`.

Four kinds, all through the public entry points:

* "op"       `multimer_attention` on ready-made projections, forward alone or forward + backward
* "combine"  `fused_multimer_combine` on materialised logits, forward + backward
* "infer"    a whole model's forward pass without gradients: logits and the last layer's representation (embedding extraction)
* "train"    a masked-language-model step: corruption, forward, loss, backward, gradients gathered into one flat buffer

Pairs are two chains `<cls> A <eos> <cls> B <eos>` of random residues, padded to T.  A pair's unpadded length is uniform in
[fill * T, T]; `skew` makes the first chain short (a peptide and its receptor) instead of splitting at 20..80 %.
"""
import math
import random

import torch

import mint_plus_b200 as M
from mint_plus_b200.distributed import FlatGradAllReduce
from mint_plus_b200.lora import apply_lora

DEV = "cuda"
# model family -> (embed, heads, head size, full depth)
MODELS = {"8m": (320, 20, 16, 6), "150m_lora": (640, 20, 32, 30), "650m_mu_fp8": (1280, 20, 64, 33), "3b_plus": (2560, 40, 64, 36)}


def _named(name, case):
    return case if name is None else dict(case, name=name)


def _op(name, B, H, T, D, dtype="bf16", grad=True, sqrt=False, fill=0.94, skew=False, meta=True):
    return _named(name, dict(kind="op", B=B, H=H, T=T, D=D, dtype=dtype, grad=grad, sqrt=sqrt, fill=fill, skew=skew, meta=meta))


def _model(name, kind, model, layers, B, T, dtype="bf16", fill=0.5, skew=False, pack=False):
    return _named(name, dict(kind=kind, model=model, layers=layers, B=B, T=T, dtype=dtype, fill=fill, skew=skew, pack=pack))


def listed():
    return [
        # one short pair through the bare operator at the 8M model's head size: latency, mask metadata built in the call
        _op("op_one_pair_d16", 1, 20, 187, 16, grad=False, meta=False),
        # the isolated-operator benchmark: the 150M head size, forward + backward
        _op("op_d32_step", 8, 20, 1024, 32),
        # the muS models' square-root softmax at the 650M head size, a length off every tile boundary, training
        _op("op_d64_sqrt_ragged_step", 5, 20, 1531, 64, sqrt=True, fill=0.5),
        # a peptide / receptor batch at the widest model's head count, inference
        _op("op_d64_skewed_fwd", 8, 40, 2048, 64, grad=False, skew=True, fill=0.45),
        # the fp32 path (reproducible runs, parity checks), training
        _op("op_fp32_d16_step", 4, 20, 401, 16, dtype="f32", fill=0.5),
        # the combine entry point for callers that hold both logit matrices
        dict(name="combine_d32_step", kind="combine", B=2, H=20, T=360, D=32, dtype="bf16"),
        # the smallest model on a CPU-sized batch in fp32
        _model("mint8m_fp32_infer", "infer", "8m", 6, 4, 512, dtype="f32", fill=0.3),
        # the same model trained in bf16 on short pairs: many short kernels
        _model("mint8m_train", "train", "8m", 6, 4, 330),
        # one pair through the FP8 650M model: serving latency
        _model("mint650m_fp8_infer_one_pair", "infer", "650m_mu_fp8", 33, 1, 497, fill=1.0),
        # a stretch of the FP8 650M training step (two layers, embedding and head) at its configured batch
        _model("mint650m_fp8_train", "train", "650m_mu_fp8", 2, 16, 2048, fill=0.1),
        # a stretch of the 150M frozen-base LoRA step at its configured batch
        _model("mint150m_lora_train", "train", "150m_lora", 8, 32, 1024, fill=0.1),
        # embedding extraction with the 36 x 2560 model on skewed pairs
        _model("mint3b_infer", "infer", "3b_plus", 36, 8, 2048, skew=True, fill=0.45),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes log-uniform between a single short pair and the configured batches."""
    what = rng.choice(["op", "op", "op", "op", "op_f32", "combine", "infer_f32", "infer_fp8", "infer_plus", "train_8m", "train_fp8", "train_lora"])
    fill, skew = rng.choice([0.1, 0.3, 0.5, 0.94, 1.0]), rng.random() < 0.3
    if what == "op":
        D = rng.choice([16, 32, 64])
        T = _log_int(rng, 64, 2048)
        H = 40 if D == 64 and rng.random() < 0.3 else 20
        B = _log_int(rng, 1, max(1, min(32, 2.7e7 // (T * T))))
        return _op(None, B, H, T, D, grad=rng.random() < 0.6, sqrt=rng.random() < 0.3, fill=fill, skew=skew, meta=rng.random() < 0.6)
    if what == "op_f32":
        T = _log_int(rng, 64, 700)
        return _op(None, _log_int(rng, 1, max(1, 1.5e6 // (T * T))), 20, T, rng.choice([16, 32]), dtype="f32", grad=rng.random() < 0.6, fill=fill,
                   skew=skew, meta=rng.random() < 0.6)
    if what == "combine":
        T = _log_int(rng, 64, 700)
        return dict(kind="combine", B=_log_int(rng, 1, max(1, min(8, 1e6 // (T * T)))), H=20, T=T, D=rng.choice([16, 32, 64]), dtype=rng.choice(["bf16", "bf16", "f32"]))
    if what == "infer_f32":
        return _model(None, "infer", "8m", 6, _log_int(rng, 1, 8), _log_int(rng, 100, 640), dtype="f32", fill=fill, skew=skew)
    if what == "infer_fp8":
        T = _log_int(rng, 100, 2048)
        return _model(None, "infer", "650m_mu_fp8", 33, _log_int(rng, 1, max(1, 16384 // T)), T, fill=fill, skew=skew, pack=rng.random() < 0.3)
    if what == "infer_plus":
        T = _log_int(rng, 100, 2048)
        return _model(None, "infer", "3b_plus", rng.choice([4, 12]), _log_int(rng, 1, max(1, 16384 // T)), T, fill=fill, skew=skew, pack=rng.random() < 0.3)
    if what == "train_8m":
        return _model(None, "train", "8m", 6, _log_int(rng, 1, 16), _log_int(rng, 64, 640), fill=fill, skew=skew)
    T = _log_int(rng, 128, 2048 if what == "train_fp8" else 1024)
    if what == "train_fp8":
        return _model(None, "train", "650m_mu_fp8", 2, _log_int(rng, 1, max(1, 32768 // T)), T, fill=fill, skew=skew, pack=rng.random() < 0.3)
    return _model(None, "train", "150m_lora", 8, _log_int(rng, 1, max(1, 32768 // T)), T, fill=fill, skew=skew)


def _pairs(case, seed):
    """(tokens, chain ids, key padding) of the batch, on the GPU."""
    r = random.Random(seed)
    B, T = case["B"], case["T"]
    tokens = torch.full((B, T), 1, dtype=torch.int64)
    chain_ids = torch.zeros(B, T, dtype=torch.int64)
    g = torch.Generator().manual_seed(seed)
    residues = torch.randint(4, 24, (B, T), generator=g)
    for b in range(B):
        n = max(8, r.randint(int(case["fill"] * T), T))
        a = min(n - 4, max(4, int(n * (r.uniform(0.02, 0.08) if case["skew"] else r.uniform(0.2, 0.8)))))
        tokens[b, :n] = residues[b, :n]
        tokens[b, 0] = tokens[b, a] = 0
        tokens[b, a - 1] = tokens[b, n - 1] = 2
        chain_ids[b, a:] = 1
    tokens, chain_ids = tokens.to(DEV), chain_ids.to(DEV)
    return tokens, chain_ids, tokens.eq(1)


def _build(case, seed):
    """The model as a user's program builds it, parameters created and initialised on the GPU."""
    torch.manual_seed(seed)
    torch.cuda.manual_seed(seed)
    E, H, _, _ = MODELS[case["model"]]
    n, kind = case["layers"], case["model"]
    with torch.device(DEV):
        if kind == "650m_mu_fp8":
            model = M.build_mint_mu("650M", num_layers=n, use_fp8=True, unit_scaled=True)
        elif kind == "3b_plus":
            model = M.MINT(num_layers=n, embed_dim=E, attention_heads=H, use_multimer=True,
                           layer_factory=lambda: M.TransformerLayer_MINT_plus(E, 4 * E, H, use_multimer=True))
        else:
            model = M.MINT(num_layers=n, embed_dim=E, attention_heads=H, use_multimer=True, use_erf_gelu=True)
    if case["dtype"] == "bf16":
        model = model.to(torch.bfloat16)
    if kind == "150m_lora":
        apply_lora(model, r=8, alpha=16.0)
        with torch.no_grad():          # adapters some steps into training: B = 0 would give A no gradient
            for name, p in model.named_parameters():
                if name.endswith("lora_B"):
                    p.normal_(0.0, 0.02)
    model.train(case["kind"] == "train")
    model.pack_padding = case["pack"]
    return model


def prepare(case, seed):
    dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    g = torch.Generator(device=DEV).manual_seed(seed)
    tokens, chain_ids, pad = _pairs({**case, "fill": case.get("fill", 0.9), "skew": case.get("skew", False)}, seed)
    s = dict(case=case)
    if case["kind"] == "op":
        shape = (case["B"], case["H"], case["T"], case["D"])
        s["qkv"] = [(torch.randn(shape, device=DEV, generator=g) / math.sqrt(case["D"])).to(dt).requires_grad_(case["grad"]) for _ in range(6)]
        s["masks"] = dict(meta=M.mask_meta_from_chain_ids(chain_ids, pad)) if case["meta"] else dict(chain_ids=chain_ids, key_padding_mask=pad)
        if case["grad"]:
            s["d_out"] = torch.randn(shape, device=DEV, generator=g).to(dt)
    elif case["kind"] == "combine":
        B, H, T, D = case["B"], case["H"], case["T"], case["D"]
        logits = [torch.randn(B, H, T, T, device=DEV, generator=g).masked_fill_(pad[:, None, None, :], float("-inf")).to(dt) for _ in range(2)]
        values = [torch.randn(B, H, T, D, device=DEV, generator=g).to(dt) for _ in range(2)]
        s["inputs"] = [t.requires_grad_(True) for t in logits + values]
        s["mask"] = chain_ids.unsqueeze(-1) != chain_ids.unsqueeze(-2)
        s["d_out"] = torch.randn(B, H, T, D, device=DEV, generator=g).to(dt)
    else:
        s["model"], s["tokens"], s["chain_ids"] = _build(case, seed), tokens, chain_ids
        if case["kind"] == "train":
            s["params"] = [p for p in s["model"].parameters() if p.requires_grad]
            s["gather"] = FlatGradAllReduce(s["params"], dtype=s["params"][0].dtype)
            s["rng"] = g
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "op":
        if not case["grad"]:
            with torch.no_grad():
                return M.multimer_attention(*s["qkv"], sqrt_softmax=case["sqrt"], **s["masks"])
        out = M.multimer_attention(*s["qkv"], sqrt_softmax=case["sqrt"], **s["masks"])
        return [out.detach(), *torch.autograd.grad(out, s["qkv"], s["d_out"])]
    if case["kind"] == "combine":
        il, el, iv, ev = s["inputs"]
        out = M.fused_multimer_combine(il, el, s["mask"], iv, ev)
        return [out.detach(), *torch.autograd.grad(out, s["inputs"], s["d_out"])]
    if case["kind"] == "infer":
        with torch.no_grad():
            out = s["model"](s["tokens"], s["chain_ids"], repr_layers=[case["layers"]])
        return [out["logits"], out["representations"][case["layers"]]]
    for p in s["params"]:
        p.grad = None
    loss, ppl = M.shared_step(s["model"], (s["tokens"], s["chain_ids"]), generator=s["rng"])
    loss.backward()
    s["gather"]()
    return [loss.detach(), ppl, s["gather"].flat]


def work(case):
    """Multiply-adds of the contractions (one logit and one value term per query and unpadded key: the pathway is selected, not
    summed) and every input, weight and result moved once."""
    B, T, size = case["B"], case["T"], 2 if case["dtype"] == "bf16" else 4
    keys = T * (1 + case.get("fill", 0.9)) / 2
    if case["kind"] == "op":
        n = B * case["H"] * T * case["D"] * size
        f = 4.0 * B * case["H"] * T * keys * case["D"]
        return {"bytes": 14.0 * n if case["grad"] else 7.0 * n, "flops": 3.5 * f if case["grad"] else f}
    if case["kind"] == "combine":
        H, D = case["H"], case["D"]
        return {"bytes": size * (4.0 * B * H * T * T + 6.0 * B * H * T * D) + B * T * T, "flops": 6.0 * B * H * T * keys * D}
    E, H, D, _ = MODELS[case["model"]]
    rows = B * keys if case["pack"] else B * T
    gemm = 30.0 * E * E * rows * case["layers"]
    attn = 4.0 * H * rows * keys * D * case["layers"]
    head = rows * (2.0 * E * E + 66.0 * E)
    weights = 15.0 * E * E * case["layers"] * (1 if case["model"] == "650m_mu_fp8" else size)
    if case["kind"] == "infer":
        return {"bytes": weights + B * T * (8 + 8 + size * (33 + E)), "flops": gemm + attn + head}
    lora = case["model"] == "150m_lora"
    out = 2 * (56.0 * E * 8 * case["layers"] if lora else 15.0 * E * E * case["layers"])
    return {"bytes": 2 * weights + B * T * 16 + out, "flops": gemm * (2 if lora else 3) + 3.5 * attn + 3 * head}


def tolerance(case):
    if case["dtype"] == "f32":
        # sums in fp32; a whole model's error grows over its layers
        return {"rel": 1e-5 if case["kind"] in ("op", "combine") else 3e-5}
    if case.get("model") == "650m_mu_fp8":
        # e4m3 activations and e5m2 gradients: a value next to a rounding boundary moves by a whole step of 6 to 25 %
        return {"rel": 0.03, "max": 0.99}
    return {"rel": 1e-2, "max": 0.99} if case["kind"] in ("train", "infer") else {"rel": 1e-2}

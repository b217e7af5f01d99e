"""The persistent attention backward at the edges of its work list, against the oracle: more items than CTAs, a key tile with more query
tiles than a ballot holds, items without a pair (padded or single-chain tiles), a last tile of one row."""
import pytest
import torch

import mint_plus_b200 as M
from oracle import multimer_attention as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,D,kind,sqrt", [
    (1, 1, 4225, 32, "pairs", False), (1, 1, 4225, 64, "pairs", True), (3, 20, 513, 16, "padded", False), (3, 20, 513, 64, "padded", False),
    (2, 40, 257, 64, "one chain", True), (1, 1, 1, 32, "one chain", False), (4, 20, 385, 32, "boundary", True)])
def test_backward_work_list(B, H, T, D, kind, sqrt):
    g = torch.Generator().manual_seed(T + D)
    ts = [torch.randn(B, H, T, D, generator=g).bfloat16().float() for _ in range(6)]
    grad = torch.randn(B, H, T, D, generator=g).bfloat16().float()
    ids = torch.zeros(B, T, dtype=torch.int64)
    pad = torch.zeros(B, T, dtype=torch.bool)
    if kind != "one chain":
        ids[:, {"pairs": T // 3, "padded": T // 5, "boundary": 128}[kind]:] = 1
    if kind == "padded":
        pad[0, 128:] = True
        pad[1, T // 2:] = True
    leaves = [t.cuda().bfloat16().requires_grad_() for t in ts]
    out = M.multimer_attention(*leaves, chain_ids=ids.cuda(), key_padding_mask=pad.cuda(), sqrt_softmax=sqrt)
    got = torch.autograd.grad(out, leaves, grad.cuda().bfloat16())
    M.check_device_status()
    kw = dict(sqrt_softmax=True) if sqrt else {}
    want_out, want = O.multimer_attention_fwd_bwd(*ts, O.chain_mask_from_ids(ids), grad, key_pad=pad, **kw)
    for a, b in zip([out.detach(), *got], [want_out, *want]):
        scale = max(b.abs().max().item(), 1e-3)
        assert (a.float().cpu() - b).abs().max().item() <= 3e-2 * scale

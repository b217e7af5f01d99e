"""The fp32 attention at the edges of its tiles (8 to 32 rows per block, 64 columns per tile), with tiles of one pathway, of both, and of
padding only, against the oracle."""
import pytest
import torch

import mint_plus_b200 as M
from oracle import multimer_attention as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sqrt_softmax", [False, True])
@pytest.mark.parametrize("T,D", [(1, 16), (31, 32), (33, 64), (64, 16), (65, 64), (127, 32), (129, 16), (200, 64), (258, 32)])
def test_fp32_attention_tile_edges(T, D, sqrt_softmax):
    B, H = 2, 3
    g = torch.Generator().manual_seed(T * 100 + D)
    ts = [torch.randn(B, H, T, D, generator=g) for _ in range(6)]
    grad = torch.randn(B, H, T, D, generator=g)
    ids = torch.zeros(B, T, dtype=torch.int64)
    ids[0, T // 2:] = 1
    ids[1, T // 3:] = 1
    ids[1, 2 * T // 3:] = 2
    pad = torch.zeros(B, T, dtype=torch.bool)
    if not sqrt_softmax:                 # (the oracle's square-root softmax has 0 * inf at padded keys)
        pad[1, T - T // 4:] = True
    if T > 100 and not sqrt_softmax:
        pad[0, 64:70] = True
    want, wg = O.multimer_attention_fwd_bwd(*ts, O.chain_mask_from_ids(ids), grad, key_pad=pad, sqrt_softmax=sqrt_softmax)
    leaves = [t.cuda().requires_grad_(True) for t in ts]
    out = M.multimer_attention(*leaves, chain_ids=ids.cuda(), key_padding_mask=pad.cuda(), sqrt_softmax=sqrt_softmax)
    got = torch.autograd.grad(out, leaves, grad.cuda())
    for a, b in zip((out, *got), (want, *wg)):
        assert (a.detach().cpu() - b).norm() <= 4e-6 * b.norm() + 3e-6

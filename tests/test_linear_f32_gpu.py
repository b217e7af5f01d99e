"""fp32 projections at the edges of their tiles (32 / 64 rows and columns, slabs of 16 to 128 columns) against float64, and the layer that
runs on them against the same layer with gradients on, whose projections are autograd's."""
import pytest
import torch

import mint_plus_b200 as M
from mint_plus_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 4, 4), (33, 36, 20), (65, 320, 132), (2048, 320, 324), (300, 1284, 320), (5120, 1288, 64)])
@pytest.mark.parametrize("gelu,res", [(False, True), (True, False)])
def test_linear_f32(m, n, k, gelu, res):
    torch.manual_seed(0)
    x, w, b = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda") * k ** -0.5, torch.randn(n, device="cuda")
    r = torch.randn(m, n, device="cuda") if res else None
    y = _lib.host().linear_f32(x, w, b, gelu, r)
    ref = x.double() @ w.double().T + b.double()
    ref = torch.nn.functional.gelu(ref) if gelu else ref + r.double()
    torch.testing.assert_close(y.double(), ref, rtol=2e-6, atol=2e-6)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("T,B,H,D", [(37, 3, 4, 16), (130, 2, 6, 32), (64, 1, 2, 64)])
def test_layer_f32(fused, T, B, H, D):
    torch.manual_seed(0)
    E = H * D
    cls = M.TransformerLayer_MINT_plus if fused else M.TransformerLayer_MINT
    layer = cls(E, 4 * E, H, use_multimer=True).cuda()
    x = torch.randn(T, B, E, device="cuda")
    chain_ids = (torch.arange(T, device="cuda") > T // 3).long().expand(B, T).contiguous()
    pad = (torch.arange(T, device="cuda") >= T - 5).expand(B, T).contiguous()
    with torch.no_grad():
        y, _ = layer(x, self_attn_padding_mask=pad, chain_ids=chain_ids)
    ref, _ = layer(x, self_attn_padding_mask=pad, chain_ids=chain_ids)
    assert ref.requires_grad
    torch.testing.assert_close(y, ref.detach(), rtol=2e-5, atol=2e-5)

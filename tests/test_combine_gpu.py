"""Combine from materialised logits at the edges of its tiles (16 query rows, 32 / 64 keys, odd and even row lengths, tensors off a
16-byte boundary) against the oracle."""
import pytest
import torch

import mint_plus_b200 as M
from oracle import multimer_attention as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,D", [(1, 16), (15, 32), (16, 64), (33, 16), (63, 64), (64, 32), (65, 64), (130, 16), (257, 32), (290, 64)])
def test_combine_tile_edges(T, D, dtype):
    B, H = 2, 3
    g = torch.Generator().manual_seed(1000 * T + D)
    il, el = (2 * torch.randn(B, H, T, T, generator=g) for _ in range(2))
    iv, ev, grad = (torch.randn(B, H, T, D, generator=g) for _ in range(3))
    mask = torch.rand(B, T, T, generator=g) < 0.5
    if T > 64:
        mask[0, :, : T // 2] = False                 # whole chunks of one pathway
        il[:, :, :, -5:] = el[:, :, :, -5:] = float("-inf")
    ts = [t.to(dtype) for t in (il, el, iv, ev, grad)]
    leaves = [t.float().requires_grad_(True) for t in ts[:4]]
    want = O.combine_from_logits(leaves[0], leaves[1], mask, leaves[2], leaves[3])
    wg = torch.autograd.grad(want, leaves, ts[4].float())
    off = [torch.empty(t.numel() + 1, dtype=dtype, device=DEV)[1:].view(t.shape).copy_(t) if D == 32 else t.to(DEV) for t in ts]
    dl = [t.requires_grad_(True) for t in off[:4]]
    out = M.fused_multimer_combine(dl[0], dl[1], mask.to(DEV), dl[2], dl[3])
    got = torch.autograd.grad(out, dl, off[4])
    tol = 2e-6 if dtype == torch.float32 else 6e-3
    for a, b in zip((out, *got), (want, *wg)):
        b = b.detach()
        assert (a.float().cpu() - b).norm() <= tol * (b.norm() + 1e-6)


def test_combine_more_than_65535_heads():
    """(batch, head) pairs beyond the 65535 blocks that a second grid dimension takes."""
    B, H, T, D = 32800, 2, 3, 16
    g = torch.Generator(DEV).manual_seed(0)
    il, el = (torch.randn(B, H, T, T, device=DEV, generator=g).requires_grad_() for _ in range(2))
    iv, ev = (torch.randn(B, H, T, D, device=DEV, generator=g).requires_grad_() for _ in range(2))
    mask = torch.rand(B, T, T, device=DEV, generator=g) < 0.5
    d = torch.randn(B, H, T, D, device=DEV, generator=g)
    out = M.fused_multimer_combine(il, el, mask, iv, ev)
    got = torch.autograd.grad(out, (il, el, iv, ev), d)
    m = mask.unsqueeze(1)
    p = torch.where(m, el, il).softmax(-1)
    want = (p * ~m) @ iv + (p * m) @ ev
    for a, b in zip((out, *got), (want, *torch.autograd.grad(want, (il, el, iv, ev), d))):
        assert (a - b).norm() <= 2e-6 * b.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("far", [False, True])
def test_combine_keeps_fp32_probabilities(dtype, far):
    """Sums whose terms cancel to about 1e-5 of their size show an error of the probabilities 1e5 times enlarged, in a bf16 result too.
    `far`: the keys that carry the values lie 40 and more below the row maximum, where a rounded exponent counts most."""
    B, H, T, D = 2, 2, 66, 16
    g = torch.Generator().manual_seed(7)
    value = torch.ones(T)
    value[1::2] = -1.0
    if far:     # two groups at logits -50 and -50 + k/8, with the bf16 value that comes closest to cancelling the first group's
        off = torch.arange(1, 81).double() / 8
        miss = (torch.exp(off) * torch.exp(-off).bfloat16().double() - 1).abs()
        k = miss.argmin()
        value[1::2] = -torch.exp(-off[k]).bfloat16().float()
        s = torch.full((B, H, T, T), -50.0)
        s[..., 1::2] += off[k].float()
        el = s.clone()
    else:
        s, el = (1e-4 * torch.randn(B, H, T, T, generator=g) for _ in range(2))
    s[..., :2] = el[..., :2] = 0.0
    value[:2] = 0.0
    v = value[:, None].expand(B, H, T, D)
    mask = ((torch.arange(T)[:, None] + torch.arange(T)[None, :] // 2) % 3 == 0).expand(B, T, T)
    il, el, iv, ev = (t.to(dtype) for t in (s, el, v, v))
    m = mask.unsqueeze(1)
    p = torch.where(m, el, il).double().softmax(-1)
    want = (p * ~m) @ iv.double() + (p * m) @ ev.double()
    size = p @ iv.double().abs()
    out = M.fused_multimer_combine(*(t.to(DEV) for t in (il, el, mask, iv, ev))).double().cpu()
    # a term is off by a few roundings of fp32: all of a group alike (far) 4 x 2^-24 at most, else some 2 x 2^-24 each, 64 of them with
    # either sign, an eighth of that in the sum; a bf16 result rounds by 2^-9 on top
    cancel = (want.norm() / size.norm()).item()
    bound = (4.0 if far else 0.25) * 2.0 ** -24 / cancel + (2.0 ** -9 if dtype == torch.bfloat16 else 0.0)
    assert (out - want).norm() <= bound * want.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("value", [float("inf"), -3.4e38])
def test_combine_infinite_and_largest_values(dtype, D, value):
    """Infinities and values at the end of the range reach the rows and dimensions that they belong to, as sums in fp32 have them."""
    B, H, T = 1, 2, 70
    g = torch.Generator().manual_seed(D)
    il, el = (torch.randn(B, H, T, T, generator=g).to(dtype) for _ in range(2))
    iv, ev, d = (torch.randn(B, H, T, D, generator=g).to(dtype) for _ in range(3))
    mask = torch.rand(B, T, T, generator=g) < 0.5
    mask[:, :20] = False
    iv[0, 0, 3, 5] = value
    ev[0, 1, T - 1, D - 1] = value
    d[0, 1, 33, 2] = value

    def exact(il, el, iv, ev, d):
        # sums over the selected elements alone, as the operator defines them
        m = mask.unsqueeze(1)
        p = torch.where(m, el, il).softmax(-1)
        sel = lambda a, keep: torch.where(keep.unsqueeze(-1), a, torch.zeros((), dtype=a.dtype))
        v = torch.where(m.unsqueeze(-1), ev.unsqueeze(-3), iv.unsqueeze(-3))              # (B,H,T,T,D): the value that (i, j) takes
        out = (p.unsqueeze(-1) * v).sum(-2)
        dp = (d.unsqueeze(-2) * v).sum(-1)
        ds = p * (dp - (p * dp).sum(-1, keepdim=True))
        g = p.unsqueeze(-1) * d.unsqueeze(-2)
        return [out, ds.masked_fill(m, 0.0), ds.masked_fill(~m, 0.0), sel(g, (~m).expand_as(p)).sum(-3), sel(g, m.expand_as(p)).sum(-3)]

    want = exact(*[t.float() for t in (il, el, iv, ev, d)])
    leaves = [t.to(DEV).requires_grad_() for t in (il, el, iv, ev)]
    out = M.fused_multimer_combine(leaves[0], leaves[1], mask.to(DEV), leaves[2], leaves[3])
    got = [out, *torch.autograd.grad(out, leaves, d.to(DEV))]
    for a, b in zip(got, want):
        b = b.to(dtype).float()                                                            # (beyond bf16's range: infinite there)
        a = a.float().cpu()
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf()) and torch.equal(a[a.isinf()], b[b.isinf()])
        f = b.isfinite()
        big = b.abs() > 1e30
        assert torch.allclose(a[f & big], b[f & big], rtol=1e-2)
        assert (a[f & ~big] - b[f & ~big]).norm() <= (2e-6 if dtype == torch.float32 else 6e-3) * b[f & ~big].norm()

"""The training step's two ends on the C++ host side: the corruption in one launch, the tied projection of an odd vocabulary."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1), (3, 85), (4, 330)])
def test_mlm_corruption_from_the_same_draws(shape):
    """The one-launch corruption against the same formula on the same draws."""
    from mint_plus_b200.training import mlm_corrupt
    tokens = torch.randint(0, 33, shape, device="cuda")
    a, b = (torch.Generator(device="cuda").manual_seed(5) for _ in range(2))
    out, target = mlm_corrupt(tokens, 0, 2, 1, 32, a)
    u, k = (torch.rand(shape, device="cuda", generator=b) for _ in range(2))
    aa = torch.randint(4, 24, shape, device="cuda", generator=b)
    want_target = (u < 0.15) & ~((tokens == 0) | (tokens == 2) | (tokens == 1))
    want = torch.where((k < 0.8) & want_target, torch.full_like(tokens, 32), tokens)
    want = torch.where((k > 0.9) & want_target, aa, want)
    assert target.dtype == torch.bool and torch.equal(target, want_target) and torch.equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 40])
@pytest.mark.parametrize("gelu", [False, True])
def test_linear_with_any_number_of_rows(n, gelu):
    """Weights whose rows are not a multiple of eight (the vocabulary): value and gradients against fp32."""
    from mint_plus_b200 import ops
    torch.manual_seed(0)
    x, w, b = (torch.randn(s, device="cuda").bfloat16().requires_grad_() for s in ((5, 7, 64), (n, 64), (n,)))
    y = ops.linear(x, w, b, gelu)
    xf, wf, bf = (t.detach().float().requires_grad_() for t in (x, w, b))
    z = xf @ wf.T + bf
    ref = torch.nn.functional.gelu(z) if gelu else z
    g = torch.randn_like(ref).bfloat16()
    assert y.shape == ref.shape
    for a, r in zip((y, *torch.autograd.grad(y, (x, w, b), g)), (ref, *torch.autograd.grad(ref, (xf, wf, bf), g.float()))):
        assert (a.float() - r).abs().max().item() <= 2e-2 * max(1.0, r.abs().max().item())

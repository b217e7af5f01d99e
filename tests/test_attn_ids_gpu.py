"""An attention call on chain ids, whose metadata and rotation are one launch, gives what the two steps give, to the bit."""
import pytest
import torch

import mint_plus_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ids_dtype,pad", [(torch.int64, True), (torch.int32, False), (torch.int16, True)])
@pytest.mark.parametrize("B,T,D,dtype,rope", [(1, 1, 16, torch.bfloat16, True), (3, 64, 32, torch.bfloat16, True), (2, 65, 64, torch.bfloat16, True),
                                              (2, 1100, 16, torch.bfloat16, True), (2, 70, 16, torch.float32, True), (2, 70, 32, torch.bfloat16, False)])
def test_ids_and_metadata_agree(B, T, D, dtype, rope, ids_dtype, pad):
    g = torch.Generator(device="cuda").manual_seed(T)
    leaves = [torch.randn(B, 3, T, D, device="cuda", generator=g).to(dtype).requires_grad_() for _ in range(6)]
    grad = torch.randn(B, 3, T, D, device="cuda", generator=g).to(dtype)
    ids = (torch.arange(T, device="cuda") > T // 3).to(ids_dtype).expand(B, T)          # not contiguous
    kpad = (torch.arange(T, device="cuda") >= T - T // 5).expand(B, T) if pad else None
    runs = []
    for kw in (dict(chain_ids=ids, key_padding_mask=kpad), dict(meta=M.mask_meta_from_chain_ids(ids, kpad))):
        out = M.multimer_attention(*leaves, rope=rope, **kw)
        runs.append([out.detach(), *torch.autograd.grad(out, leaves, grad)])
    M.check_device_status()
    for i, (a, b) in enumerate(zip(*runs)):
        if dtype == torch.bfloat16 and i in (1, 4):       # dQ: its additions have no fixed order
            assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()
        else:
            assert torch.equal(a, b)
    with pytest.raises(ValueError):
        M.multimer_attention(*leaves, rope=rope, chain_ids=ids[:, : T - 1] if T > 1 else ids.expand(B + 1, T), key_padding_mask=None)

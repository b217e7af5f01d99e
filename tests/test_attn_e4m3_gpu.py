"""The e4m3 copy that the attention forward leaves of its result is the quantisation of that result, to the bit."""
import pytest
import torch

import mint_plus_b200 as M
from mint_plus_b200 import _lib as L, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sqrt_softmax,seq_first", [(False, True), (True, False)])
@pytest.mark.parametrize("B,T,D", [(1, 1, 16), (3, 127, 32), (2, 129, 64), (2, 300, 16)])
def test_copy_is_the_quantised_result(B, T, D, sqrt_softmax, seq_first):
    H, scale = 3, 0.25
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = [torch.randn(B, H, T, D, device="cuda", generator=g).bfloat16() for _ in range(6)]
    qkv[2], qkv[5] = qkv[2] * 200, qkv[5] * 1e-3                         # beyond 448 / scale, and subnormal
    ids = (torch.arange(T, device="cuda") > T // 2).long().expand(B, T)
    pad = torch.zeros(B, T, dtype=torch.bool, device="cuda")
    if B > 1:
        pad[-1] = True                                                   # nothing but padding: NaN rows
    meta = M.mask_meta_from_chain_ids(ids, pad)
    flags = (L.FLAG_SQRT_SOFTMAX if sqrt_softmax else 0) | (L.FLAG_OUT_SEQ_FIRST if seq_first else 0)
    out = torch.empty((T, B, H, D) if seq_first else (B, H, T, D), device="cuda", dtype=torch.bfloat16)
    out8 = torch.zeros(out.shape, device="cuda", dtype=torch.uint8)
    lse = torch.empty(B, H, T, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = L.lib().mintb_attn_fwd_e4m3(*(t.data_ptr() for t in qkv), meta.buf.data_ptr(), None, None, out.data_ptr(), lse.data_ptr(), None, 0, B, H, T, D, flags,
                                     D ** -0.5, out8.data_ptr(), 1 / scale, torch.cuda.current_stream().cuda_stream, status.data_ptr())
    assert rc == L.OK and status.item() == 0
    ref = M.multimer_attention(*qkv, meta=meta, rope=False, sqrt_softmax=sqrt_softmax, out_seq_first=seq_first)
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16).view(out.shape))
    assert torch.equal(out8, ops.quantize_e4m3(out, scale).view(torch.uint8))
    if B > 1:
        assert out.isnan().any()

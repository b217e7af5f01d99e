"""Projections on CTA pairs (256 x 256 tiles of two SMs) against the fp32 product of the same operands: ragged rows and columns, a pair
whose second half holds no row, both operand types, with and without the activation."""
import pytest
import torch

from mint_plus_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bf16", "e4m3"])
@pytest.mark.parametrize("M,N,K", [(2500, 2008, 5136), (2432, 2304, 4096), (4609, 1288, 5120), (18945, 256, 4112)])
@pytest.mark.parametrize("gelu", [0, 1])
def test_linear_on_cta_pairs(dtype, M, N, K, gelu):
    torch.manual_seed(0)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float8_e4m3fn
    x = torch.randn(M, K, device="cuda").to(dt)
    w = (torch.randn(N, K, device="cuda") / 8).to(dt)
    bias = torch.randn(N, device="cuda")
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib = _lib.lib()
    rc = lib.mintb_linear_fwd(x.data_ptr(), w.data_ptr(), bias.data_ptr(), out.data_ptr(), None, M, N, K,
                              _lib.BF16 if dtype == "bf16" else _lib.E4M3, _lib.F32, _lib.BF16, gelu, 0.125, 1.0,
                              torch.cuda.current_stream().cuda_stream, status.data_ptr())
    assert rc == 0, lib.mintb_last_error()
    ref = 0.125 * (x.float() @ w.float().T) + bias
    if gelu:
        ref = torch.nn.functional.gelu(ref)
    assert status.item() == 0
    assert (out.float() - ref).abs().max().item() <= 6e-3 * ref.abs().max().item()

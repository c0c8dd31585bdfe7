"""GEMM epilogue on outputs whose rows are not 16-byte aligned, and the staged bias, at tile edges."""

import pytest
import torch

import iree_turbine_b200 as tb
from iree_turbine_b200 import ops
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


# n % 8: 1 and 3 -> 2-byte stores (4-byte for fp32), 2 -> 4-byte, 4 -> 8-byte; one column, one past a
# piece, a tile edge -1 / +1, several tiles; m = 1, a partial and a full 32-row band
@pytest.mark.parametrize("m,n", [(1, 1), (33, 65), (130, 127), (97, 129), (256, 258), (31, 260), (300, 515), (700, 1203)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_unaligned_output_rows(m, n, out_dtype):
    a, b = oracle.make_gemm_inputs(m, n, 72, torch.bfloat16, seed=31)
    ref = oracle.gemm_nt(a, b)
    c = torch.ops.b200k.gemm_nt(a.to(DEV), b.to(DEV), out_dtype)
    oracle.assert_close_half(c, ref)
    # a bias on the same sizes: exact against the plain result, since fp32 out = acc + bias rounds once
    bias = torch.randn(n, generator=torch.Generator().manual_seed(32))
    y = torch.ops.b200k.linear_act(a.to(DEV), b.to(DEV), bias.to(DEV), "none", out_dtype)
    torch.cuda.synchronize()
    assert tb.device_status() == 0
    if out_dtype == torch.float32:
        assert torch.equal(y, c + bias.to(DEV))
    else:
        oracle.assert_close_half(y, ref + bias)


# whole tiles with one epilogue (bias none: the values come through the product), with the other, and split-K
@pytest.mark.parametrize("n,k,split", [(200, 64, 1), (1203, 8, 1), (200, 512, 2)])
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16])
def test_silu_over_the_whole_range(n, k, split, bias_dtype):
    low = torch.finfo(bias_dtype).min
    x = torch.cat([torch.tensor([0.0, -0.0, 1.0, 20.0, 88.0, 104.0, 3e38, -20.0, -86.9, -87.4, -88.6, -88.8, -100.0, -1e4, -1e30, -1e36,
                                 low, low / 2, 1e-30, -1e-30]), torch.linspace(-95, 95, n - 23)])
    x = torch.cat([x, torch.tensor([float("inf"), -float("inf"), float("nan")])]).to(bias_dtype)
    a, w = torch.zeros(3, k, dtype=torch.bfloat16, device=DEV), torch.zeros(n, k, dtype=torch.bfloat16, device=DEV)
    out = torch.full((3, n), 7.0, device=DEV)
    ops._launch_gemm(a, w, out, None, None, bias=x.to(DEV), activation="silu", split_k=split)
    got, x64 = out.cpu().double(), x.double()
    assert tb.device_status() == 0 and torch.equal(got[1].nan_to_num(), got[0].nan_to_num())
    ref = x64 / (1.0 + torch.exp(-x64))
    # the exponential is good to 2 + 1.173 |x| units of 2^-23, the sum and the quotient to one each; e^-x overflows
    # beyond 88.7, where the exact result is below 3e-37 and a zero is due
    finite = x64.isfinite()
    bound = (4 + 1.173 * x64.abs().clamp(max=104)) * 2.0 ** -23 * ref.abs() + 3e-37
    assert bool(((got[0] - ref).abs() <= bound)[finite].all())
    assert got[0, -3] == float("inf") and bool(got[0, -2:].isnan().all())


# n ends 2 to 14 bytes into a 16-byte piece of a row whose pitch is a multiple of 16 bytes
@pytest.mark.parametrize("n,ldc", [(6, 8), (33, 40), (130, 136), (515, 520)])
@pytest.mark.parametrize("dtype,out_dtype", [(torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("tile_m,tile_n", [(128, 64), (128, 128), (128, 256), (256, 256)])
def test_columns_past_n_are_not_written(n, ldc, dtype, out_dtype, tile_m, tile_n):
    a, b = oracle.make_gemm_inputs(150, n, 136, dtype, seed=51)
    c = torch.full((150, ldc), 7.0, dtype=out_dtype, device=DEV)
    ops._launch_gemm(a.to(DEV), b.to(DEV), c[:, :n], None, None, tile_m=tile_m, tile_n=tile_n, split_k=1)
    assert bool((c[:, n:] == 7.0).all())
    oracle.assert_close_half(c[:, :n], oracle.gemm_nt(a, b), rtol=2e-2, atol=2e-2)

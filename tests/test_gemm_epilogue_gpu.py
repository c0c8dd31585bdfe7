"""GEMM epilogue on outputs whose rows are not 16-byte aligned, and the staged bias, at tile edges."""

import pytest
import torch

import iree_turbine_b200 as tb
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

"""The GEMM that stores its column shard into every rank's matrix, with one rank: shards of less than a tile."""

import ctypes as C

import pytest
import torch

import iree_turbine_b200 as tb
from iree_turbine_b200 import _launcher as L
from iree_turbine_b200 import ops
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 8 columns are the 16 bytes a shard has at least; both sides of 64 and of 128 columns
@pytest.mark.parametrize("n", [8, 40, 64, 72, 128, 136])
@pytest.mark.parametrize("m", [5, 300])
@pytest.mark.parametrize("plain", [0, 1])
def test_narrow_shards(m, n, plain):
    k, offset = 200, 16
    a, b = oracle.make_gemm_inputs(m, n, k, torch.bfloat16, seed=37)
    ad, bd = a.to(DEV), b.to(DEV)
    full = torch.full((m, offset + n + 8), -7.0, dtype=torch.bfloat16, device=DEV)
    g = L.GemmAllGatherArgs()
    g.gemm.a, g.gemm.b = ad.data_ptr(), bd.data_ptr()
    g.gemm.m, g.gemm.n, g.gemm.k, g.gemm.lda, g.gemm.ldb = m, n, k, k, k
    g.gemm.in_dtype = g.gemm.out_dtype = L.DTYPE_CODES[torch.bfloat16]
    g.gemm.status = ops._status_ptr(full.device)
    g.peer_c[0] = full.data_ptr()
    g.num_peers, g.peer_ldc, g.col_offset, g.plain_stores = 1, full.stride(0), offset, plain
    L.check(L.lib().b200k_gemm_nt_allgather(C.byref(g), ops._stream(full)))
    torch.cuda.synchronize()
    assert tb.device_status() == 0
    oracle.assert_close_half(full[:, offset:offset + n], oracle.gemm_nt(a, b))
    assert bool((full[:, :offset] == -7).all()) and bool((full[:, offset + n:] == -7).all())

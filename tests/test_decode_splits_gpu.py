"""How the decode kernel splits a history: one chunk, clusters of 2 / 4 / 8, a second kernel; ring depths."""

import pytest
import torch

import iree_turbine_b200 as tb
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (sequences, q heads, kv heads, longest history, chunk): chunk 0 = the library's rule.  Histories include
# 0, 1 and the longest; the chunk counts are 1, 2, 3, 5, 8 (clusters, whose last CTAs have nothing to do for
# the short ones), 9 and 36 (second kernel, one and several batches per warp); the units below and above
# one wave of CTAs; 16 heads per group and 1.
@pytest.mark.parametrize("seqs,hq,hkv,longest,chunk", [
    (3, 16, 1, 64, 0), (3, 4, 4, 128, 0), (4, 8, 2, 129, 64), (4, 8, 2, 190, 64), (3, 32, 2, 320, 64), (5, 8, 2, 512, 64),
    (4, 8, 8, 576, 64), (2, 8, 2, 2304, 64), (40, 8, 8, 300, 0), (3, 8, 4, 2500, 0), (2, 16, 1, 5000, 0), (160, 2, 2, 200, 64),
])
@pytest.mark.parametrize("dim", [128, 64])
def test_every_split_matches_the_oracle(seqs, hq, hkv, longest, chunk, dim):
    lens = [longest, 0, 1] + [(7919 * i) % (longest + 1) for i in range(3, seqs)]
    q, kc, vc, bt, sl = oracle.make_paged_decode_inputs(q_heads=hq, kv_heads=hkv, head_dim=dim, lens=lens[:seqs], seed=41)
    scale = dim ** -0.5
    got = torch.ops.b200k.paged_decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), scale, chunk)
    again = torch.ops.b200k.paged_decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), scale, chunk)
    torch.cuda.synchronize()
    assert tb.device_status() == 0
    oracle.assert_close_half(got.cpu(), oracle.paged_decode_attention(q, kc, vc, bt, sl, scale))
    assert torch.equal(got, again)
    if seqs > 1:
        assert torch.equal(got[1].cpu(), torch.zeros(hq, dim, dtype=q.dtype))


@pytest.mark.parametrize("chunk", [64, 512])
@pytest.mark.parametrize("dim", [128, 64])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_the_largest_probability_of_every_tile_is_exact(chunk, dim, dtype):
    """One key of every 16 counts (the others' weights are below e^-50): its 16-bit probability is 1 whatever the chunk is,
    so the result is the 64-bit one, rounded once.  Scores carry 2^-22 each, exponentials as much and the fp32 sums
    of 32 tiles 2^-21: 4e-6 decides nothing but a value that close to the middle between two 16-bit ones."""
    g = torch.Generator().manual_seed(43)
    seqs, hq, hkv, length = 3, 4, 2, 512
    k = torch.zeros(seqs, hkv, length, dim)
    k[..., 0] = -60.0
    for tile in range(length // 16):
        k[:, :, tile * 16 + (5 * tile) % 16, 0] = -3.0 * torch.rand(seqs, hkv, generator=g)
    v = 1.0 + torch.rand(seqs, hkv, length, dim, generator=g)
    k, v = k.to(dtype), v.to(dtype)
    q = torch.zeros(seqs, hq, dim, dtype=dtype)
    q[..., 0] = 1.0
    lens = torch.full((seqs,), length, dtype=torch.int32)
    got = torch.ops.b200k.decode_attention(q.to(DEV), k.to(DEV), v.to(DEV), lens.to(DEV), 1.0, chunk).cpu()
    p = torch.softmax(k[..., 0].double(), -1)
    ref = torch.einsum("skt,sktd->skd", p, v.double()).repeat_interleave(hq // hkv, 1)
    near = (ref * (1 - 4e-6)).to(dtype) != (ref * (1 + 4e-6)).to(dtype)
    assert near.float().mean() < 0.05
    assert torch.equal(got[~near], ref.to(dtype)[~near])

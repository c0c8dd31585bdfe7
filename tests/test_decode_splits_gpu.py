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


def split_chunk(units, capacity, length):
    """Tokens per chunk where the rule is "about 400 CTAs of at least 192 tokens": by the length, not by the capacity."""
    n = -(-400 // units)
    return 2048 if length > 2048 * n else max(192, -(-(-(-length // n)) // 64) * 64)


# (sequences, kv heads, capacity, lengths): tables and caches with room for more than the histories in them.  8 units
# with a cluster rule for the capacity, 8 and 32 units with the other, 160 and 320 units; lengths of 0 and 1
# token, around a chunk and around 2048 times the number of chunks, and the capacity itself.
@pytest.mark.parametrize("seqs,hkv,capacity,lens", [
    (1, 8, 2048, [1000]), (4, 8, 4096, [100, 0, 1500, 4096]), (1, 8, 131072, [1000]), (4, 8, 131072, [191, 192, 193, 2500]),
    (4, 8, 32768, [1, 0, 32768, 1000]), (20, 8, 8192, [8192, 2048, 2049, 0] + [300] * 16), (40, 8, 16384, [2047, 2048, 2049, 4097, 0] + [100] * 35),
])
@pytest.mark.parametrize("paged", [True, False])
def test_capacity_above_the_lengths(seqs, hkv, capacity, lens, paged):
    q, kc, vc, bt, sl = oracle.make_paged_decode_inputs(q_heads=2 * hkv, kv_heads=hkv, head_dim=64, lens=lens, seed=44)
    if not paged and seqs * hkv * capacity > 1 << 22:
        pytest.skip("the table form covers it")
    ref = oracle.paged_decode_attention(q, kc, vc, bt, sl, 0.125)
    q, sl = q.to(DEV), sl.to(DEV)
    if paged:
        table = torch.zeros(seqs, capacity // 16, dtype=torch.int32)
        table[:, :bt.shape[1]] = bt.clamp(min=0)
        rest = (kc.to(DEV), vc.to(DEV), table.to(DEV), sl, 0.125)
        op = torch.ops.b200k.paged_decode_attention
    else:
        rest = tuple(torch.ops.b200k.paged_gather(c.to(DEV), bt.to(DEV), sl, capacity) for c in (kc, vc)) + (sl, 0.125)
        op = torch.ops.b200k.decode_attention
    got = op(q, *rest)
    torch.cuda.synchronize()
    assert tb.device_status() == 0
    oracle.assert_close_half(got.cpu(), ref)
    assert torch.equal(got, op(q, *rest))
    units = seqs * hkv
    if units < 296 and capacity > 4096:  # the same bits as with every sequence's chunk asked for by hand
        for s, n in enumerate(lens):
            assert torch.equal(got[s], op(q, *rest, split_chunk(units, capacity, n))[s]), (s, n)


@pytest.mark.parametrize("chunk", [64, 512, 0])  # second kernel, cluster, one chunk
def test_rows_without_a_positive_sum_are_zero(chunk):
    """Scores that are all -infinity or NaN give zeros, infinite values or not; the other rows are untouched."""
    seqs, length, dim = 3, 640 if chunk else 64, 128
    k = torch.randn(seqs, 2, length, dim, generator=torch.Generator().manual_seed(45)).half()
    v = torch.randn(seqs, 2, length, dim, generator=torch.Generator().manual_seed(46)).half()
    q = torch.randn(seqs, 4, dim, generator=torch.Generator().manual_seed(47)).half()
    lens = torch.full((seqs,), length, dtype=torch.int32)
    ref = oracle.decode_attention(q, k, v, lens, 0.1)
    q[0], k[0], v[0] = 1.0, -float("inf"), float("inf")
    q[1] = float("nan")
    got = torch.ops.b200k.decode_attention(q.to(DEV), k.to(DEV), v.to(DEV), lens.to(DEV), 0.1, chunk).cpu()
    assert torch.equal(got[:2], torch.zeros(2, 4, dim, dtype=torch.float16))
    oracle.assert_close_half(got[2], ref[2])

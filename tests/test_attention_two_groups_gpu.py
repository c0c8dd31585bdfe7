"""Head dim 64, long items: a query tile has two softmax warpgroups that take its half steps of 64 keys in turn.

Keys from 1536 on average run there (paged: and 1536 queries), so sizes are odd and even counts of half steps around it; the
ramp makes the running max grow by more than 2^8 in half steps of either warpgroup, so that both rescale the accumulator and
each other's sums.
"""

import pytest
import torch

import iree_turbine_b200 as tb

pytestmark = pytest.mark.gpu
DEV = "cuda"


def normal(shape, seed, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def check(got, q, k, v, scale, offset, dtype):
    """One head against 64 bits: probabilities and output are rounded to 16 bits once each."""
    s = (q.double() @ k.double().t()) * scale
    if offset is not None:
        s.masked_fill_(~torch.ones_like(s, dtype=torch.bool).tril(offset), -torch.inf)
    p = torch.softmax(s, -1).nan_to_num(0.0)
    ref = p @ v.double()
    eps = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -11
    bound = 2 * eps * (p @ v.double().abs() + ref.abs()) + 1e-4
    assert bool(((got.double() - ref).abs() <= bound).all())
    return torch.logsumexp(s, -1)


@pytest.mark.parametrize("b,h,hkv,sq,skv", [(1, 2, 1, 1, 1536), (2, 3, 3, 300, 1537), (1, 2, 2, 129, 1700), (1, 160, 8, 257, 1792),
                                            (1, 1, 1, 3100, 3100)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("ramp", [False, True])
def test_dense(b, h, hkv, sq, skv, causal, dtype, ramp):
    q, k, v = normal((b, h, sq, 64), 1, dtype), normal((b, hkv, skv, 64), 2, dtype), normal((b, hkv, skv, 64), 3, dtype)
    if ramp:
        k = k * torch.linspace(0.1, 6.0, skv, device=DEV, dtype=dtype)[:, None]
    got, lse = torch.ops.b200k.attention_lse(q, k, v, 0.3, causal)
    for i, j in {(0, 0), (b - 1, h - 1)}:
        kj = j // (h // hkv)
        want = check(got[i, j], q[i, j], k[i, kj], v[i, kj], 0.3, skv - sq if causal else None, dtype)
        # fp32 scores of up to 64 products of a few units each, and a sum of positive terms
        assert bool(((lse[i, j].double() - want).abs() <= 1e-4 * (1 + want.abs())).all())
        one = torch.ops.b200k.attention(q[i:i + 1, j:j + 1], k[i:i + 1, kj:kj + 1], v[i:i + 1, kj:kj + 1], 0.3, causal)
        assert torch.equal(got[i, j], one[0, 0])  # whatever the CTA did before
    assert tb.device_status() == 0


@pytest.mark.parametrize("skv", [64, 100, 128, 129, 300, 1700])
@pytest.mark.parametrize("first,last", [(0, 64), (64, 128), (0, 10000), (10, 11)])
def test_nan_keys(skv, first, last):
    """A NaN among the keys reaches output and statistic of every row, whichever half steps it is in."""
    q, k, v = (normal((1, 2, s, 64), i, torch.bfloat16) for i, s in enumerate((5, skv, skv)))
    k[:, :, first:last] = float("nan")
    out, lse = torch.ops.b200k.attention_lse(q, k, v, 0.1, False)
    if first < skv:
        assert bool(out.isnan().all()) and not bool(lse.isfinite().any())
    else:
        assert bool(out.isfinite().all()) and bool(lse.isfinite().all())
    assert tb.device_status() == 0


@pytest.mark.parametrize("page", [16, 128])
@pytest.mark.parametrize("sq", [200, 1600])  # one warpgroup per tile, two
def test_paged(page, sq):
    lens, h, hkv = [3000, 65, 0, 1601, 2990], 4, 2
    counts = [-(-n // page) for n in lens]
    perm = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(5)).to(torch.int32)
    table = torch.zeros((len(lens), max(counts)), dtype=torch.int32)
    for row, part in zip(table, perm.split(counts)):
        row[: part.numel()] = part
    dtype = torch.bfloat16
    kc, vc = (normal((sum(counts), hkv, page, 64), s, dtype) for s in (1, 2))
    q = normal((len(lens), h, sq, 64), 3, dtype)
    got = torch.ops.b200k.paged_attention(q, kc, vc, table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), 0.3, True)
    for i, n in enumerate(lens):
        pages = table[i, : counts[i]].long().to(DEV)
        for j in range(h):
            k, v = (c[pages, j // 2].reshape(-1, 64)[:n] for c in (kc, vc))
            check(got[i, j], q[i, j], k, v, 0.3, n - sq, dtype)
    assert tb.device_status() == 0

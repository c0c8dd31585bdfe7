"""Item orders of the attention forward kernels: every item is done once, whatever the list looks like.

A head's result does not depend on which CTA computed it or on what else was in the call, so the whole call
must equal, bit for bit, calls on one head (or one sequence) at a time, whose lists are a single round.
"""

import pytest
import torch

import iree_turbine_b200 as tb
from iree_turbine_b200 import _launcher as L
from iree_turbine_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
KERNELS = [L.ATTN_ONE_TILE, L.ATTN_TILE_PAIR]


@pytest.fixture(autouse=True)
def automatic_kernel():
    yield
    ops.ATTENTION_KERNEL = L.ATTN_AUTO


def normal(shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.bfloat16)


# (batch, heads, kv heads, queries, keys): less than a round; a last round that is partly full, in an odd and in
# an even round; one item per head; couples with a middle pair of its own and rounds filled to 95 %; rows that
# see no key; heads in groups, the last one smaller (K/V beyond what L2 shares)
@pytest.mark.parametrize("b,h,hkv,sq,skv", [(1, 3, 3, 300, 300), (2, 40, 8, 520, 520), (5, 37, 37, 300, 300), (3, 100, 4, 90, 90),
                                            (1, 74, 2, 900, 900), (1, 148, 4, 640, 700), (2, 50, 2, 600, 200),
                                            (1, 56, 56, 4000, 4000)])
@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("causal", [True, False])
def test_dense_order(b, h, hkv, sq, skv, kernel, causal):
    q, k, v = normal((b, h, sq, 128), 1), normal((b, hkv, skv, 128), 2), normal((b, hkv, skv, 128), 3)
    ops.ATTENTION_KERNEL = kernel
    got = torch.ops.b200k.attention(q, k, v, 0.1, causal)
    for i in range(b):
        for j in range(h):
            kj = j // (h // hkv)
            one = torch.ops.b200k.attention(q[i:i + 1, j:j + 1], k[i:i + 1, kj:kj + 1], v[i:i + 1, kj:kj + 1], 0.1, causal)
            assert torch.equal(got[i, j], one[0, 0])
    scores = (q[0, -1].double() @ k[0, -1].double().t()) * 0.1
    if causal:
        scores.masked_fill_(~torch.ones(sq, skv, dtype=torch.bool, device=DEV).tril(skv - sq), -torch.inf)
    ref = torch.softmax(scores, -1).nan_to_num(0.0) @ v[0, -1].double()  # rows that see no key give zeros
    # probabilities and output rounded to bf16 (2^-9 each, relative): of sums of |v|, all below 8
    bound = 2.0 ** -9 * (torch.softmax(scores, -1).nan_to_num(0.0) @ v[0, -1].double().abs() + ref.abs()) + 1e-3
    assert bool(((got[0, -1].double() - ref).abs() <= bound).all())
    assert tb.device_status() == 0


# (lengths, queries, heads, kv heads): equal lengths; an empty sequence and one shorter than its queries; more
# rounds than one; more (sequence, tile) entries than are sorted
@pytest.mark.parametrize("lens,sq,h,hkv", [([700] * 3, 300, 4, 2), ([1000, 0, 100, 513], 257, 6, 6), ([90, 2000, 700, 1500, 10], 400, 64, 2),
                                           ([(37 * i) % 400 for i in range(530)], 17, 2, 1)])
@pytest.mark.parametrize("kernel", KERNELS + [L.ATTN_AUTO])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dim", [128, 64])
def test_paged_order(lens, sq, h, hkv, kernel, causal, dim):
    page = 32
    counts = [max(1, -(-n // page)) for n in lens]
    order = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(4)).int()
    table = torch.zeros(len(lens), max(counts), dtype=torch.int32)
    for row, part in zip(table, order.split(counts)):
        row[:part.numel()] = part
    table, sl = table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    kc, vc, q = normal((sum(counts), hkv, page, dim), 5), normal((sum(counts), hkv, page, dim), 6), normal((len(lens), h, sq, dim), 7)
    ops.ATTENTION_KERNEL = kernel
    got = torch.ops.b200k.paged_attention(q, kc, vc, table, sl, 0.1, causal)
    for i in range(0, len(lens), max(1, len(lens) // 8)):
        if dim == 64 or kernel != L.ATTN_AUTO:  # AUTO may take another kernel for one sequence
            one = torch.ops.b200k.paged_attention(q[i:i + 1], kc, vc, table[i:i + 1], sl[i:i + 1], 0.1, causal)
            assert torch.equal(got[i], one[0])
        n = lens[i]
        if n == 0:
            assert not got[i].any()
            continue
        k = torch.ops.b200k.paged_gather(kc, table[i:i + 1], sl[i:i + 1], n)
        v = torch.ops.b200k.paged_gather(vc, table[i:i + 1], sl[i:i + 1], n)
        dense = torch.ops.b200k.attention(q[i:i + 1], k, v, 0.1, causal)[0]
        if dim == 64 or kernel != L.ATTN_AUTO:
            assert torch.equal(dense, got[i])
        else:  # the two kernels round the probabilities to bf16 against different running maxima (2^-8 of |v| < 8)
            assert torch.allclose(dense.float(), got[i].float(), rtol=2.0 ** -7, atol=2.0 ** -5)
    assert tb.device_status() == 0

"""One-tile kernel: steps of 64 keys that three softmax warpgroups take in turn, over items of every length."""
import pytest
import torch

import iree_turbine_b200 as tb
from iree_turbine_b200 import _launcher as L
from iree_turbine_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def automatic_kernel():
    yield
    ops.ATTENTION_KERNEL = L.ATTN_AUTO


def normal(shape, seed, dtype=torch.float16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def check(q, k, v, scale, causal, got):
    s = q.double() @ k.double().transpose(2, 3) * scale
    if causal:
        s.masked_fill_(~torch.ones(s.shape[2:], dtype=torch.bool, device=DEV).tril(k.size(2) - q.size(2)), -torch.inf)
    p = torch.softmax(s, -1).nan_to_num(0.0)
    ref = p @ v.double()
    # one rounding of each probability, one of the output (2^-11 each, relative)
    assert bool(((got.double() - ref).abs() <= 2.0 ** -11 * (p @ v.double().abs() + ref.abs()) + 1e-4).all())
    assert tb.device_status() == 0


# 1 to 7 steps, whole and partly masked, an odd last half of a tile; 600 items: CTAs start items with any of the warpgroups
@pytest.mark.parametrize("skv", [1, 63, 64, 65, 127, 128, 129, 192, 193, 257, 385, 448])
@pytest.mark.parametrize("causal", [False, True])
def test_steps(skv, causal):
    q, k, v = normal((4, 75, 200, 128), 1), normal((4, 75, skv, 128), 2), normal((4, 75, skv, 128), 3)
    ops.ATTENTION_KERNEL = L.ATTN_ONE_TILE
    got = torch.ops.b200k.attention(q, k, v, 0.1, causal)
    check(q, k, v, 0.1, causal, got)
    assert torch.equal(got[-1:, -1:], torch.ops.b200k.attention(q[-1:, -1:], k[-1:, -1:], v[-1:, -1:], 0.1, causal))


# The running maximum rises by more than 2^8 in every step, in some, and in the last one: each time the accumulator is rescaled
# between the products of two other warpgroups
@pytest.mark.parametrize("rises", ["every", "third", "last"])
def test_rescaling(rises):
    n = 1000
    q, k, v = normal((2, 40, 256, 128), 1), normal((2, 40, n, 128), 2), normal((2, 40, n, 128), 3)
    step = torch.arange(n, device=DEV) // 64
    height = {"every": step, "third": step // 3, "last": step // 15}[rises].half() * (20.0 if rises != "last" else 300.0)
    q[..., 0], k[..., 0] = 10.0, height  # adds up to 200 (3000) * scale per step to the scores
    ops.ATTENTION_KERNEL = L.ATTN_ONE_TILE
    for _ in range(3):
        got = torch.ops.b200k.attention(q, k, v, 0.1, False)
        check(q, k, v, 0.1, False, got)

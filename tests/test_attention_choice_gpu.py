"""Which forward kernel a call gets (``B200K_ATTN_AUTO``)."""

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


def normal(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


# Query tiles that fill two or four rounds over 148 SMs, pairs of them one or two; one round of either; a single head.
@pytest.mark.parametrize("b,h,hkv,sq,skv", [(1, 37, 37, 1000, 300), (4, 32, 8, 512, 512), (2, 74, 2, 257, 1000), (1, 3, 1, 700, 900)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_without_a_mask_the_kernel_does_not_depend_on_the_batch(b, h, hkv, sq, skv, dtype):
    """Head dim 128 without a mask is the one-tile kernel's, so a head has the bits of a call on that head alone."""
    q, k, v = normal((b, h, sq, 128), 1, dtype), normal((b, hkv, skv, 128), 2, dtype), normal((b, hkv, skv, 128), 3, dtype)
    got = torch.ops.b200k.attention(q, k, v, 0.1, False)
    for i, j in {(0, 0), (b - 1, h - 1)}:
        kj = j // (h // hkv)
        one = torch.ops.b200k.attention(q[i:i + 1, j:j + 1], k[i:i + 1, kj:kj + 1], v[i:i + 1, kj:kj + 1], 0.1, False)
        assert torch.equal(got[i, j], one[0, 0])
    ops.ATTENTION_KERNEL = L.ATTN_ONE_TILE
    assert torch.equal(got, torch.ops.b200k.attention(q, k, v, 0.1, False))
    assert tb.device_status() == 0

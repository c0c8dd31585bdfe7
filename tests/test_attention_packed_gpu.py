"""Head dim 64, one query tile and one K/V tile per head, more heads than SMs: two heads per item."""
import pytest
import torch

import iree_turbine_b200 as tb

pytestmark = pytest.mark.gpu
DEV = "cuda"


def normal(shape, seed, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


# one head more than SMs and an odd count; several rounds; a grouped K/V head; one row, one key, one and two half steps; rows that
# see no key; nothing visible but to the last row
@pytest.mark.parametrize("b,h,hkv,sq,skv", [(1, 149, 149, 128, 128), (32, 8, 8, 128, 128), (15, 40, 5, 100, 64), (3, 75, 25, 1, 1),
                                            (5, 61, 61, 17, 65), (7, 32, 8, 128, 3), (2, 90, 90, 3, 128), (2, 100, 100, 128, 1)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_two_heads_per_item(b, h, hkv, sq, skv, causal, dtype):
    """Each head has the bits of a call on it alone, in its own rows and nowhere else."""
    q, k, v = normal((b, h, sq, 64), 1, dtype), normal((b, hkv, skv, 64), 2, dtype), normal((b, hkv, skv, 64), 3, dtype)
    got, lse = torch.ops.b200k.attention_lse(q, k, v, 0.125, causal)
    group = h // hkv
    s = q.double() @ k.double().repeat_interleave(group, 1).transpose(2, 3) * 0.125
    if causal:
        s.masked_fill_(~torch.ones(sq, skv, dtype=torch.bool, device=DEV).tril(skv - sq), -torch.inf)
    p, vv = torch.softmax(s, -1).nan_to_num(0.0), v.double().repeat_interleave(group, 1)
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8  # one rounding of each probability, one of the output
    assert bool(((got.double() - p @ vv).abs() <= eps * (p @ vv.abs() + (p @ vv).abs()) + 1e-6).all())
    ref = torch.logsumexp(s, -1)
    assert torch.equal(torch.isinf(lse), torch.isinf(ref))
    assert torch.allclose(lse.double().nan_to_num(neginf=0.0), ref.nan_to_num(neginf=0.0), rtol=1e-5, atol=1e-4)
    for i, j in ((0, 0), (0, 1), (b - 1, h - 1), (b // 2, h // 2)):
        one, one_lse = torch.ops.b200k.attention_lse(q[i:i + 1, j:j + 1], k[i:i + 1, j // group:j // group + 1],
                                                     v[i:i + 1, j // group:j // group + 1], 0.125, causal)
        assert torch.equal(got[i, j], one[0, 0]) and torch.equal(lse[i, j], one_lse[0, 0])
    assert tb.device_status() == 0

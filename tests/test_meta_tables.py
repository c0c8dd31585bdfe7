"""Meta implementations take what the CUDA ones take (torch.compile traces through them): tables, lengths, positions and
histories of more sequences than the call's, and column vectors; too few and other types are refused."""

import pytest
import torch

from iree_turbine_b200 import ops  # noqa: F401  (registers the operators)

OP = torch.ops.b200k


def empty(*shape, dtype=torch.float16):
    return torch.empty(shape, dtype=dtype, device="meta")


def table(rows, dtype=torch.int32):
    return empty(rows, 8, dtype=dtype)


def vector(*shape, dtype=torch.int32):
    return empty(*shape, dtype=dtype)


CACHE = empty(20, 2, 16, 128)
CALLS = {
    "paged_decode": lambda t, n: OP.paged_decode_attention(empty(3, 4, 128), CACHE, CACHE, t, n, 0.1),
    "paged_attention": lambda t, n: OP.paged_attention(empty(3, 4, 5, 128), CACHE, CACHE, t, n, 0.1, True),
    "paged_gather": lambda t, n: OP.paged_gather(CACHE, t, n, 100),
    "kv_append": lambda t, n: OP.kv_append(empty(3, 5, 2, 128), empty(3, 5, 2, 128), CACHE, CACHE, t, n),
    "decode": lambda t, n: OP.decode_attention(empty(3, 4, 128), empty(t.size(0), 2, 50, 128), empty(t.size(0), 2, 50, 128), n, 0.1),
}


@pytest.mark.parametrize("name", CALLS)
def test_same_calls_as_on_the_device(name):
    fn = CALLS[name]
    for lens in (vector(3), vector(5), vector(3, 1), vector(1, 3)):
        fn(table(3), lens)
    out = fn(table(5), vector(5))
    if name != "kv_append":
        assert out.size(0) == (5 if name == "paged_gather" else 3)
    for lens in (vector(2), vector(3, 2), vector(3, dtype=torch.int64)):
        with pytest.raises(RuntimeError, match="must be int32"):
            fn(table(3), lens)
    if name != "decode":
        with pytest.raises(RuntimeError, match="must be int32"):
            fn(table(3, dtype=torch.int64), vector(3))
    if name != "paged_gather":  # whose number of sequences is the table's
        with pytest.raises(RuntimeError, match="block_table must be|one history per sequence"):
            fn(table(2), vector(3))


def test_dense_attention_takes_keys_of_more_sequences():
    assert OP.attention(empty(2, 4, 7, 128), empty(3, 2, 9, 128), empty(3, 2, 9, 128), 0.1, False).shape == (2, 4, 7, 128)
    with pytest.raises(RuntimeError, match="batch mismatch"):
        OP.attention(empty(4, 4, 7, 128), empty(3, 2, 9, 128), empty(3, 2, 9, 128), 0.1, False)

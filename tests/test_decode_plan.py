"""The split of a decode call on the CPU: whatever the length, its chunks fit the grid and the workspace of the capacity."""

import ctypes as C

import pytest

from iree_turbine_b200 import _launcher as L

SMS = 148  # also what the library assumes without a GPU


def plan(lib, seqs, kv_heads, capacity):
    a = L.DecodeArgs()
    a.num_seqs, a.q_heads, a.kv_heads, a.head_dim, a.max_seq_len = seqs, kv_heads, kv_heads, 128, capacity
    per_chunk = seqs * kv_heads * (128 * 4 + 8)
    size = lib.b200k_decode_workspace_bytes(C.byref(a))
    assert size % per_chunk == 0
    return size // per_chunk, lib.b200k_decode_default_chunk(C.byref(a))


def rule(units, capacity):
    """(parts a history is split into, least tokens per part), restated; 0 parts: chunks of that many tokens."""
    slots = 2 * SMS
    if units >= slots or capacity <= 128 or (units * 4 >= slots and capacity <= 1024):
        return 0, -(-(-(-capacity // -(-capacity // 2048))) // 64) * 64
    c = 1
    while c < 8 and units * c * 2 <= SMS and c * 64 < capacity:
        c *= 2
    if c < 8 and units * c * 2 <= slots and capacity > c * 512:
        c *= 2
    return (c, 64) if capacity <= c * 512 else (-(-400 // units), 192)


def chunk(length, split, least):
    if split == 0:
        return least
    return 2048 if length > 2048 * split else max(least, -(-(-(-length // split)) // 64) * 64)


@pytest.mark.parametrize("seqs,kv_heads", [(1, 1), (1, 8), (3, 1), (4, 8), (9, 8), (10, 8), (37, 1), (74, 1), (75, 1), (37, 8), (64, 8), (128, 16)])
def test_chunks_of_every_length_fit(kernel_lib, seqs, kv_heads):
    for capacity in (1, 64, 128, 129, 512, 1000, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 16000, 40000, 131072):
        slots, given = plan(kernel_lib, seqs, kv_heads, capacity)
        split, least = rule(seqs * kv_heads, capacity)
        assert given == chunk(capacity, split, least)
        for length in {*range(0, min(capacity, 5000) + 1, 37), *range(max(0, capacity - 70), capacity + 1), 2047, 2048, 2049, 4095, 4097}:
            if length <= capacity:
                c = chunk(length, split, least)
                assert c % 64 == 0 and c <= 2048 and -(-length // c) <= slots, (capacity, length, c, slots)

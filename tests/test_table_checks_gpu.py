"""Block tables, lengths and positions of the paged and decode operators: what is refused on the host and what is taken."""

import pytest
import torch

import iree_turbine_b200 as tb
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"
OP = torch.ops.b200k
LENS = [40, 7, 100]


@pytest.fixture
def calls():
    """Operator calls with their table and their per-sequence vector left open, and the CPU inputs behind them."""
    q, kc, vc, bt, sl = oracle.make_paged_decode_inputs(q_heads=4, kv_heads=2, lens=LENS, seed=51)
    dq, dk, dv = q.to(DEV), kc.to(DEV), vc.to(DEV)
    new = torch.randn(3, 5, 2, 128, generator=torch.Generator().manual_seed(52)).half().to(DEV)
    q4 = torch.randn(3, 4, 5, 128, generator=torch.Generator().manual_seed(53)).half().to(DEV)
    contiguous = [OP.paged_gather(c, bt.to(DEV), sl.to(DEV), 112) for c in (dk, dv)]
    return {
        "paged_decode": lambda t, n: OP.paged_decode_attention(dq, dk, dv, t, n, 0.1),
        "paged_attention": lambda t, n: OP.paged_attention(q4, dk, dv, t, n, 0.1, True),
        "paged_gather": lambda t, n: OP.paged_gather(dk, t, n, 112),
        "kv_append": lambda t, n: (lambda k, v: (OP.kv_append(new, new, k, v, t, n - 5), k)[1])(dk.clone(), dv.clone()),
        "decode": lambda t, n: OP.decode_attention(dq, *contiguous, n, 0.1),
    }, bt.to(DEV), sl.to(DEV)


@pytest.mark.parametrize("name", ["paged_decode", "paged_attention", "paged_gather", "kv_append", "decode"])
def test_wrong_types_and_too_few_rows_are_refused(calls, name):
    fns, bt, sl = calls
    fn = fns[name]
    if name != "decode":
        for table in (bt.long(), bt.float(), bt[0], bt[None]):
            with pytest.raises(RuntimeError, match="block_table must be int32"):
                fn(table, sl)
        if name != "paged_gather":  # whose number of sequences is the table's
            with pytest.raises(RuntimeError, match="block_table must be int32"):
                fn(bt[:2], sl)
    for lens in (sl.long(), sl.float(), sl[:2], sl.repeat(2, 2)):
        with pytest.raises(RuntimeError, match="must be int32"):
            fn(bt, lens)
    torch.cuda.synchronize()
    assert tb.device_status() == 0


@pytest.mark.parametrize("name", ["paged_decode", "paged_attention", "paged_gather", "kv_append", "decode"])
def test_rows_of_more_sequences_and_column_vectors_are_taken(calls, name):
    fns, bt, sl = calls
    fn = fns[name]
    ref = fn(bt, sl)
    more = torch.cat([bt, bt.flip(0)])
    lens = torch.cat([sl, sl])
    table = bt if name == "paged_gather" else more
    assert torch.equal(fn(table, lens), ref)
    assert torch.equal(fn(bt, sl[:, None]), ref) and torch.equal(fn(bt, sl[None]), ref)
    assert torch.equal(fn(bt.repeat(1, 2)[:, :bt.shape[1]], sl), ref)  # a table that is a slice of a wider one
    assert tb.device_status() == 0


def test_gather_stops_where_a_table_row_ends():
    _, kc, _, bt, _ = oracle.make_paged_decode_inputs(q_heads=4, kv_heads=2, lens=[32, 32], seed=54)
    lens = torch.tensor([100, 20], dtype=torch.int32)
    got = OP.paged_gather(kc.to(DEV), bt.to(DEV), lens.to(DEV), 128).cpu()
    ref = oracle.paged_gather(kc, bt, torch.tensor([32, 20], dtype=torch.int32), 128)
    assert torch.equal(got, ref)


def test_dense_attention_takes_keys_of_more_sequences():
    q, k, v = oracle.make_attention_inputs(3, 4, 2, 70, 90, 128, torch.float16, seed=55)
    q, k, v = q[:2].to(DEV), k.to(DEV), v.to(DEV)
    assert torch.equal(OP.attention(q, k, v, 0.1, False), OP.attention(q, k[:2], v[:2], 0.1, False))
    decode = OP.decode_attention(q[:, :, 0].contiguous(), k, v, torch.tensor([90, 40, 3], dtype=torch.int32, device=DEV), 0.1)
    oracle.assert_close_half(decode, oracle.decode_attention(q[:, :, 0].cpu(), k[:2].cpu(), v[:2].cpu(),
                                                             torch.tensor([90, 40], dtype=torch.int32), 0.1))

"""How decode attention cuts a step's tokens (ops/cuda_ops.py: CudaOps.attention): what a captured step does must not depend on how long
the engine's sequences may become."""
import types

import pytest
import torch

from phaseshift_b200.ops import cuda_ops
from phaseshift_b200.ops.cuda_ops import CudaOps
from phaseshift_b200.ops.specs import AttnSpec

HQ, HKV, D = 8, 4, 64


def launch(monkeypatch, kv_fmt, rows, multi, static, max_seq_len, visible, n_seqs=0):
    """(launcher, its split length or None) of a step's first attention launch."""
    calls = []
    monkeypatch.setattr(cuda_ops._lib, "call", lambda name, *args: calls.append((name, [getattr(x, "value", None) for x in args])))
    o = object.__new__(CudaOps)
    o.device, o.ws, o.checked, o.step_rows, o.step_bucket, o.launches = torch.device("cpu"), {}, False, 0, 0, 0
    o.act_dtype, o.exact_rows, o.attn_decode_tc, o.sms, o.split_tokens = torch.bfloat16, False, True, 148, 64
    while -(-(max_seq_len + 1) // o.split_tokens) > 512:
        o.split_tokens *= 2
    o.max_splits = -(-(max_seq_len + 1) // o.split_tokens)
    t = torch.zeros(1)
    st = types.SimpleNamespace(kv_fmt=kv_fmt, kv_fp8=kv_fmt == 1, block_table=t, max_blocks=1, num_pages=1, status=t, sc=types.SimpleNamespace(page_tokens=16))
    b = types.SimpleNamespace(graph_static=static, several_rows=multi, row_pos=t, row_pos_short=t, row_slot=t, seq_desc=t, max_seqs=16,
                              n_seqs=n_seqs or (1 if multi else rows), seqs=[types.SimpleNamespace(token_ids=[0] * (rows if multi else 1))])
    kv = types.SimpleNamespace(k=t, v=torch.zeros(1), k_scale=t, v_scale=t)
    buf = o.buf
    o.buf = lambda name, r, c, dtype=torch.bfloat16: buf(name, r, 1, dtype)          # (only addresses are used)
    o.attention(torch.zeros(rows, HQ * D), AttnSpec(HQ, HKV, D, 1.0), b, kv, st, max_seq_len + 1 if static else visible)
    name, args = calls[0]
    return name, None if name == "ps_attn_decode_tc_even" else args[-6], o


@pytest.mark.parametrize("max_seq_len", [2000, 32767, 32768, 131072, 1 << 20])
@pytest.mark.parametrize("rows,multi", [(9, True), (16, True), (16, False), (64, False)])
def test_even_shares_whatever_the_longest_context(monkeypatch, max_seq_len, rows, multi):
    name, _, o = launch(monkeypatch, 0, rows, multi, True, max_seq_len, 0)
    # a (sequence, KV head) is shared by at most one CTA per tile of 64 tokens, and by at most one per SM
    assert name == "ps_attn_decode_tc_even" and o.max_splits >= min(-(-(max_seq_len + 1) // 64), o.sms)


@pytest.mark.parametrize("max_seq_len", [2000, 131072])
def test_captured_rows_of_one_sequence_have_a_fixed_length(monkeypatch, max_seq_len):
    name, split, o = launch(monkeypatch, 2, 16, True, True, max_seq_len, 0)
    assert name == "ps_paged_attention_fp4" and split == max(256, o.split_tokens)
    # batches of single rows, captured or not, and steps outside of a graph have a few CTAs per SM in all
    want = (4 * 148) // (16 * HKV)
    assert launch(monkeypatch, 2, 16, False, True, max_seq_len, 0)[1] == max(o.split_tokens, -(-(-(-(max_seq_len + 1) // want)) // 32) * 32)
    assert launch(monkeypatch, 2, 16, True, False, max_seq_len, 1500)[1] == max(o.split_tokens, -(-(-(-1500 // want)) // 32) * 32)
    assert launch(monkeypatch, 2, 8, True, True, max_seq_len, 0)[1] == o.split_tokens


def test_few_splits_are_kept_outside_of_a_graph(monkeypatch):
    """One wave of splits that are no longer than a share and a few tiles needs no shares; anything else has them."""
    assert launch(monkeypatch, 0, 16, True, False, 20000, 2000)[0] == "ps_attn_decode_tc_ex"           # 8 splits x 4 heads
    assert launch(monkeypatch, 0, 16, False, False, 20000, 2000)[0] == "ps_attn_decode_tc_even"        # 8 x 4 x 16 sequences
    # a few single rows beside a long prompt: rows and with them the splits' length are the prompt's
    assert launch(monkeypatch, 0, 800, False, False, 20000, 2500, n_seqs=16)[0] == "ps_attn_decode_tc_even"
    assert launch(monkeypatch, 0, 16, True, False, 20000, 18000)[0] == "ps_attn_decode_tc_even"        # 32 tiles a split, 8 a share


def test_rows_of_a_step_that_share_their_preparation():
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    b = StepBatch(16, 4, torch.device("cpu"), pinned=False)
    for rows, several, many in (([1], False, False), ([1, 1, 1], False, False), ([2], True, False), ([3, 3], True, False), ([4], True, True), ([5, 3], True, True)):
        b.fill([SeqRows(i, 0, [0] * n, ()) for i, n in enumerate(rows)])
        assert (b.several_rows, b.multi_rows) == (several, many), rows

"""A step's packed description (runtime/batch.py, filled by the host runtime) against a plain loop over its requests."""
import random

import numpy as np
import pytest
import torch

from phaseshift_b200.runtime.batch import SAMPLING_ROW_DTYPE, SeqRows, StepBatch


def _plain(mr, ms, short, seqs):
    a = np.zeros(5 * mr + 4 * ms, dtype=np.int32)
    a[mr:3 * mr] = -1
    pshort = 4 * mr + 4 * ms
    a[pshort:] = -1
    samp, r, visible = [], 0, 1
    for i, s in enumerate(seqs):
        n = len(s.token_ids)
        a[r:r + n] = [int(t) for t in s.token_ids]
        a[mr + r:mr + r + n] = s.slot
        pos = np.arange(s.pos_start, s.pos_start + n)
        a[2 * mr + r:2 * mr + r + n] = pos
        a[pshort + r:pshort + r + n] = pos if n <= short else -2
        a[3 * mr + 4 * i:3 * mr + 4 * i + 4] = (r, n, s.slot, s.pos_start)
        for j, o in enumerate(s.output_rows):
            a[3 * mr + 4 * ms + len(samp)] = r + o
            samp.append((1 if s.temperature <= 0.0 else 2, s.temperature, s.top_p, s.top_k, s.seed, s.sample_index + j))
        visible, r = max(visible, s.pos_start + n), r + n
    outs = a[3 * mr + 4 * ms:3 * mr + 4 * ms + len(samp)]
    return a, np.array(samp, dtype=SAMPLING_ROW_DTYPE), r, visible, len(samp) == r and list(outs) == list(range(r))


def test_fill_matches_a_loop_over_the_requests():
    rng = random.Random(3)
    for _ in range(400):
        mr, ms = rng.choice((1, 2, 8, 64, 256)), rng.choice((1, 3, 16))
        b = StepBatch(mr, ms, torch.device("cpu"))
        for _ in range(2):                                   # the second fill finds the first one's values
            seqs, left = [], mr
            for i in range(rng.randint(0, ms)):
                n = rng.choice((0, 1, 1, 2, rng.randint(0, 40)))
                if n > left:
                    break
                left -= n
                ids = [rng.randint(0, 200000) for _ in range(n)]
                ids = rng.choice((ids, tuple(ids), np.array(ids, dtype=np.int64), torch.tensor(ids, dtype=torch.int64)))
                outs = sorted(rng.sample(range(n), rng.randint(0, n)))
                seqs.append(SeqRows(i, rng.randint(0, 5000), ids, rng.choice((outs, tuple(outs), range(n))), rng.choice((0.0, 0.7, -1.0)), rng.random(),
                                    rng.randint(0, 50), rng.getrandbits(64), rng.randint(0, 99)))
            b.fill(seqs)
            ints, samp, rows, visible, identity = _plain(mr, ms, b.SHORT_SEQ_ROWS, seqs)
            assert np.array_equal(b.h_int.numpy(), ints) and np.array_equal(b._np_samp[:len(samp)], samp)
            assert (b.n_rows, b.n_seqs, b.n_out, b.max_visible, b.identity_out) == (rows, len(seqs), len(samp), visible, identity)
            b.upload()
            assert torch.equal(b.d_int, b.h_int) and torch.equal(b.d_samp, b.h_samp)


@pytest.mark.parametrize("seqs,error", [([SeqRows(0, 0, [1]), SeqRows(1, 0, [1]), SeqRows(2, 0, [1])], ValueError),
                                        ([SeqRows(0, 0, [1] * 9)], ValueError), ([SeqRows(0, 0, [1 << 40])], OverflowError),
                                        ([SeqRows(0, 0, [1], (0,), seed=-1)], OverflowError), ([SeqRows(0, 0, ["a"])], TypeError)])
def test_fill_refuses(seqs, error):
    with pytest.raises(error):
        StepBatch(8, 2, torch.device("cpu")).fill(seqs)


def test_fill_takes_numbers_as_an_integer_array_takes_them():
    """Floats and texts are cut and read, numpy's integers keep their low bits, and a row may end at the last position of 32 bits."""
    b = StepBatch(8, 4, torch.device("cpu"))
    b.fill([SeqRows(1.0, 3.0, [1.0, 2.7, "7"], [1.0], temperature=np.float32(0.5), top_k=20.0, seed=5.0, sample_index=4.0),
            SeqRows(np.int64(2), np.int64(9), np.array([4, 2 ** 32 + 5], dtype=np.int64), torch.tensor([1]), top_k=np.int64(-1), seed=np.int64(-2)),
            SeqRows(0, 2 ** 31 - 1, torch.tensor([6]), (x for x in [0])), SeqRows(0, 0, np.array([3.0], dtype=np.float32))])
    a = b.h_int.numpy()
    assert a[:7].tolist() == [1, 2, 7, 4, 5, 6, 3] and a[8:15].tolist() == [1, 1, 1, 2, 2, 0, 0]
    assert a[16:23].tolist() == [3, 4, 5, 9, 10, 2 ** 31 - 1, 0] and b.n_out == 3
    s = b._np_samp
    assert [int(x) for x in s["top_k"][:2]] == [20, 2 ** 32 - 1] and [int(x) for x in s["seed"][:2]] == [5, 2 ** 64 - 2] and int(s["sample_index"][0]) == 4


@pytest.mark.parametrize("seqs,error", [([SeqRows(0, 0, [1, 2], (0, 1), sample_index=2 ** 64 - 1)], OverflowError), ([SeqRows(0, 2 ** 31 - 1, [1, 2])], OverflowError),
                                        ([SeqRows(0, 0, (x for x in [1, 2]), (0,))], TypeError), ([SeqRows(0, 0, {1, 2}, (0,))], TypeError),
                                        ([SeqRows(0, 0, {1: 2}, (0,))], TypeError), ([SeqRows(0, 0, b"ab", (0,))], ValueError),
                                        ([SeqRows(0, 0, torch.ones(2, 1, dtype=torch.int64), (0,))], ValueError), ([SeqRows(0, 0, [np.ones(1)], (0,))], TypeError)])
def test_fill_refuses_what_is_no_row_of_numbers(seqs, error):
    with pytest.raises(error):
        StepBatch(8, 4, torch.device("cpu")).fill(seqs)

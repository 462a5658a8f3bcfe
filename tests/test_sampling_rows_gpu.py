"""Sampling with rows shared by the CTAs of a cluster (csrc/kernels/sampling.cu) against the host's draws: vocabularies and row counts that
give clusters of 8, 4, 2 and 1; ties, masks, failures and rejected attempts whose deciding token belongs to any of the CTAs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sampler():
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.ops.cuda_ops import CudaOps
    return CudaOps(tiny_config(), torch.device("cuda:0"))


def _batch(rows):
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    b = StepBatch(len(rows), len(rows), torch.device("cuda:0"))
    b.fill([SeqRows(0, 0, [0], (0,), **r) for r in rows])
    return b


# cluster sizes: 8, 8, 4 | 8 | 4 | 2, 2 | 1
@pytest.mark.parametrize("V,n", [(151936, 5), (40001, 30), (40001, 40), (32768, 2), (16387, 9), (8195, 6), (8192, 7), (8192, 160)])
def test_rows_match_the_host(V, n):
    from phaseshift_b200.utils.sampling import sample_row_host
    g = torch.Generator(device="cuda").manual_seed(V + n)
    logits = torch.randn(n, V, device="cuda", generator=g) * 3
    kinds = [dict(), dict(temperature=1.0, seed=5, sample_index=3), dict(temperature=0.7, top_k=20, seed=6, sample_index=1), dict(temperature=1.3, top_p=0.8, seed=7),
             dict(temperature=1.0, top_p=0.9, top_k=50, seed=8), dict(temperature=0.4, top_p=0.05, seed=9), dict(temperature=1.0, top_k=1, seed=10)]
    rows = [dict(kinds[i % len(kinds)]) for i in range(n)]
    for i, r in enumerate(rows):
        if r:
            r["seed"] = r["seed"] + 100 * i
    b = _batch(rows)
    none = n - 1
    b._np_samp[none]["mode"] = 0
    b.upload()
    words = (V + 31) // 32
    mask = torch.randint(-2 ** 31, 2 ** 31, (n, words), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
    active = (torch.arange(n, device="cuda") % 3 == 1).to(torch.uint8)
    ops = _sampler()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.sample(logits, b, n, mask=mask, mask_active=active, status=status).cpu().tolist()
    lg, mk = logits.cpu(), mask.cpu().numpy().view(np.uint32)
    for r in range(n if V < 100000 else min(n, 5)):
        assert got[r] == sample_row_host(lg[r], b._np_samp[r], mk[r] if int(active[r]) else None), (r, rows[r])
    assert got[none] == -1 and int(status[0]) == 0


@pytest.mark.parametrize("V,size", [(151936, 8), (16387, 4), (8195, 2)])
def test_ties_masks_and_failures_in_any_share(V, size):
    ops = _sampler()
    per = 1024 * (4 if V % 4 == 0 else 1)                        # neighbouring tokens that a CTA reads before the next one's
    later, wrapped, last = per + 3, per * size + 1, V - 1        # in the second CTA's share; in the first one's second round; the last token
    base = torch.randn(8, V, generator=torch.Generator().manual_seed(V)) * 2
    base[0, 2] = base[0, later] = 40.0                           # ties go to the lower id, whichever CTA has it
    base[1, later] = base[1, wrapped] = 40.0
    base[2, last] = 40.0
    hot = dict(temperature=1.0, top_p=0.5, seed=3)
    b = _batch([dict(), dict(), dict(), dict(), dict(temperature=1.0, seed=1), dict(), hot, dict()])
    b.upload()
    mask = torch.full((8, (V + 31) // 32), -1, dtype=torch.int32)
    for r, tok in ((3, later), (4, last)):                       # one token left, outside of the first share
        mask[r] = 0
        mask[r, tok // 32] = np.array(1 << (tok % 32), dtype=np.uint32).astype(np.int32).item()
    mask[5] = 0                                                  # none left
    base[6, later] = 60.0                                        # all of the mass
    active = torch.ones(8, dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    run = lambda x: ops.sample(x.cuda(), b, 8, mask=mask.cuda(), mask_active=active, status=status).cpu().tolist()
    got = run(base)
    assert got[:7] == [2, later, last, later, last, -1, later] and got[7] == int(base[7].argmax()) and int(status[0]) == 0
    for tok in (0, later, wrapped, last):
        for bad in (float("nan"), float("inf"), float("-inf")):
            x = base.clone()
            x[7, tok] = bad
            status.zero_()
            again = run(x)
            assert again[7] == -1 and again[:7] == got[:7] and int(status[0]) == 4


def test_more_rows_than_a_grid_has_lines():
    ops, n = _sampler(), 70000
    b = _batch([dict()])
    b.upload()
    b.d_samp = b.d_samp[:b._np_samp.dtype.itemsize].repeat(n)
    logits = torch.randn(n, 8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert torch.equal(ops.sample(logits, b, n, status=status).long(), logits.argmax(1)) and int(status[0]) == 0

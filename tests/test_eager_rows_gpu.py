"""Steps outside of a graph compute the rows they have, in the buffers of their row bucket."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(family):
    from phaseshift_b200.models import registry
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import build_engine_weights, random_getter
    from phaseshift_b200.runtime.engine import Engine
    from phaseshift_b200.runtime.state import StateConfig
    dev = torch.device("cuda:0")
    w = (registry.random_weights(registry.preset_config("gebuzen-tiny"), dev, dtype=torch.bfloat16) if family == "gebuzen"
         else build_engine_weights(tiny_config(), random_getter(tiny_config(), 0, dev), family, dev))
    return Engine(w, dev, StateConfig(max_slots=3, max_seq_len=640, page_tokens=16))


@pytest.mark.parametrize("family", ["bf16", "nvfp4", "gebuzen"])
def test_rows_of_a_step_are_as_in_its_bucket(family):
    from phaseshift_b200.runtime.batch import SeqRows
    eng = _engine(family)
    runner = type(eng.runner)
    assert runner.any_rows
    eng.apply_block_updates([(s, b, 1 + 40 * s + b) for s in range(3) for b in range(40)])
    ids = torch.randint(0, 200, (600,), generator=torch.Generator().manual_seed(0)).tolist()
    sizes = ((17,), (33, 1), (65, 2, 1), (130,), (257, 17), (515, 1))
    got = {}
    for any_rows in (True, False):
        eng.runner.any_rows = any_rows
        for lens in sizes:
            for s in range(3):
                eng.state.reset_slot(s)
            rows = [SeqRows(s, 0, ids[s:s + n], range(n)) for s, n in enumerate(lens)]
            _, out, status = eng.run_rows(rows, want_logits=True)
            assert status == 0
            got.setdefault(lens, []).append(out.logits.double().clone())
    for lens, (a, b) in got.items():
        # what depends on the number of rows of a step is the order of 32-bit sums, seen through a few layers of bf16 (or 4-bit) activations
        assert a.shape == b.shape and float((a - b).norm() / b.norm()) < 3e-2, lens


def test_steps_of_one_bucket_share_buffers():
    from phaseshift_b200.runtime.batch import SeqRows
    eng = _engine("bf16")
    eng.apply_block_updates([(0, b, 1 + b) for b in range(40)])
    for n in (512, 300, 511, 257, 400):
        eng.state.reset_slot(0)
        eng.run_rows([SeqRows(0, 0, list(range(n)), (n - 1,))])
    whole = {k[0]: t.data_ptr() for k, t in eng.ops.ws.items() if k[1] == 512}
    parts = {k: t for k, t in eng.ops.ws.items() if 256 < k[1] < 512}
    assert {k[1] for k in parts} == {272, 304, 400} and all(t.data_ptr() == whole[k[0]] and t.shape[0] == k[1] for k, t in parts.items())

"""Graph capture and the cycle collector (utils/graphs.py): off while a capture runs, as it was afterwards, and not run for it."""
import contextlib
import gc

import pytest
import torch

from phaseshift_b200.utils import graphs


@pytest.mark.parametrize("enabled", [True, False])
@pytest.mark.parametrize("fails", [False, True])
def test_collector_is_off_during_a_capture_and_not_run_before_it(monkeypatch, enabled, fails):
    collected = []

    @contextlib.contextmanager
    def graph(g, stream=None):
        yield
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: "graph")
    monkeypatch.setattr(torch.cuda, "Stream", lambda device: None)
    monkeypatch.setattr(torch.cuda, "graph", graph)
    monkeypatch.setattr(gc, "collect", lambda *a: collected.append(a))

    def step():
        assert not gc.isenabled()
        if fails:
            raise RuntimeError("a launch that cannot be captured")
        return "out"
    was = gc.isenabled()
    (gc.enable if enabled else gc.disable)()
    try:
        if fails:
            with pytest.raises(RuntimeError):
                graphs.capture("cuda:0", step)
        else:
            assert graphs.capture("cuda:0", step) == ("graph", "out")
        assert gc.isenabled() == enabled and not collected
    finally:
        (gc.enable if was else gc.disable)()

"""How many rows a step outside of a graph computes (runtime/engine.py: Engine._eager_rows)."""
from types import SimpleNamespace

import pytest

from phaseshift_b200.runtime.batch import resolve_row_bucket
from phaseshift_b200.runtime.engine import Engine


@pytest.mark.parametrize("n", [1, 2, 3, 9, 16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 1499, 2047, 2048])
def test_rows_of_an_eager_step(n):
    def rows(backend="cuda", any_rows=True, tp=None):
        bucket = resolve_row_bucket(n)
        return Engine._eager_rows(SimpleNamespace(backend=backend, runner=SimpleNamespace(any_rows=any_rows), tp=tp, EAGER_ROW_STEP=16), n, bucket), bucket
    run, bucket = rows()
    assert n <= run <= bucket and (run == bucket or (run % 16 == 0 and run - n < 16))
    # the thresholds of kernel selection are buckets, so none lies between the rows and their bucket
    assert resolve_row_bucket(run) == bucket
    assert rows(backend="ref")[0] == n
    assert rows(any_rows=False)[0] == rows(tp=SimpleNamespace(size=2))[0] == bucket
    assert rows(tp=SimpleNamespace(size=1))[0] == run

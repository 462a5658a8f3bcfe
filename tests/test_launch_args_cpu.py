"""Arguments of the kernel launchers."""
import ctypes

import numpy as np
import pytest

from phaseshift_b200.ops import _lib


def test_cached_integers_are_what_ctypes_makes_of_a_value():
    for v in (4, 0, -1, 1, 2 ** 31 - 1):
        assert _lib.c_int(v) is _lib.c_int(v) and _lib.c_int(v).value == v
    assert _lib.c_int(np.int64(4)).value == 4 and _lib.c_int(True).value == 1
    for v in (4.0, np.float32(1.0), "4", None):
        with pytest.raises(TypeError):
            ctypes.c_int(v)
        with pytest.raises(TypeError):
            _lib.c_int(v)

"""Token lists on their way into the engine: what ctypes makes of them, whichever way they go."""
import ctypes as C

import numpy as np
import pytest

from vllm_tgis_adapter_b200.engine.core import _int32_array


@pytest.mark.parametrize("values", [
    [], (), [5], (5, 6), list(range(3000)), [0, 2**31 - 1, -(2**31)], [2**31, -(2**31) - 1, 2**40 + 3, 1], [True, False],
    [C.c_int32(7), 8], [8, 2**40, C.c_int32(7)], [np.int64(3), np.int32(4)], np.arange(5, dtype=np.int32), range(4)])
def test_entries(values):
    got, want = _int32_array(values), (C.c_int32 * len(values))(*values)
    assert type(got) is type(want) and list(got) == list(want)


@pytest.mark.parametrize("values", [[1.0], [None], ["1"], [C.c_int64(7)], [1, 2.5]])
def test_refusals(values):
    with pytest.raises(TypeError) as want:
        (C.c_int32 * len(values))(*values)
    with pytest.raises(TypeError) as got:
        _int32_array(values)
    assert str(got.value) == str(want.value)


def test_the_array_keeps_its_memory():
    arrays = [_int32_array([i] * 64) for i in range(200)]
    assert all(list(a) == [i] * 64 for i, a in enumerate(arrays))

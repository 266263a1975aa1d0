"""Lists of numbers written natively into the arrays that the kernels read: what numpy would write, and nothing taken that it refuses."""

import numpy as np
import pytest


def _written(numbers, n=None):
    from qwen25vl_lite.ops.host import host_ints
    n = len(numbers) if n is None else n
    out = np.full(len(numbers) + 8, -7, dtype=np.int32)
    ok = host_ints(numbers, n, out.ctypes.data + 16)
    assert (out[:4] == -7).all() and (out[4 + n:] == -7).all()
    return ok, out[4:4 + n]


class _Index:
    def __init__(self, value, then=None):
        self.value, self.then = value, then

    def __index__(self):
        if self.then:
            self.then()
        return self.value


@pytest.mark.parametrize("numbers", [[], [5], [0, -1, 2 ** 31 - 1, -2 ** 31], list(range(1000)), [np.int64(4), np.int32(-3), True, _Index(9)]])
def test_lists_are_written_as_numpy_writes_them(numbers):
    ok, out = _written(numbers)
    assert ok and out.tolist() == [int(np.int64(x)) if not isinstance(x, _Index) else x.value for x in numbers]


@pytest.mark.parametrize("numbers", [[1, 2 ** 31], [-2 ** 31 - 1], [1, 10 ** 30], [1.0], ["1"], [None]])
def test_what_is_no_32_bit_int_is_left_to_the_caller(numbers):
    assert not _written(numbers)[0]


def test_a_list_of_another_length_is_left_to_the_caller():
    assert not _written([1, 2, 3], 2)[0]
    numbers = [1, 2, 3]
    numbers[0] = _Index(1, numbers.clear)
    assert not _written(numbers)[0]

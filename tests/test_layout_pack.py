"""Layout.to_c takes what a ctypes array of three ints takes, with its results and its errors:
short lists are filled with zeros (which the library refuses), integers are taken modulo 2^32, and
everything else raises ctypes' own exception."""
import ctypes as C

import numpy as np
import pytest

from bricklib_gb300 import _abi, bricks as B

GIVEN = [(8, 8, 8), [8, 8, 8], np.array([8, 4, 2]), (True, 8, 8), (np.int32(8),) * 3, (C.c_int(8), 8, 8),
         (8, 8), (8, 8, 8, 8), (), (2 ** 32 + 8, 8, 8), (2 ** 31, 8, -1), (8.0, 8, 8), ("8", 8, 8), (None, 8, 8), 8, None]


def outcome(f):
    try:
        return bytes(f())
    except Exception as e:  # noqa: BLE001
        return type(e)


@pytest.mark.parametrize("given", GIVEN, ids=repr)
@pytest.mark.parametrize("field", ["bdim", "fold"])
def test_layout_to_c_is_a_ctypes_array_of_three(field, given):
    one = (8, 8, 8)
    want = outcome(lambda: _abi.bk_layout((C.c_int * 3)(*(given if field == "bdim" else one)),
                                          (C.c_int * 3)(*(given if field == "fold" else one))))
    assert outcome(lambda: B.Layout(**{"bdim": one, "fold": one, field: given}).to_c()) == want

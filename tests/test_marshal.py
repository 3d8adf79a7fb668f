"""The structs' row pointers (marshal.py): each member at its row of the block, and a block of another height."""
import ctypes

import numpy as np
import pytest

from pypo_gb300 import Structs as S
from pypo_gb300 import marshal as M

ROWS = ("x", "y", "z", "nx", "ny", "nz", "area")


@pytest.mark.parametrize("ctype", [ctypes.c_float, ctypes.c_double])
def test_container_members_are_the_rows(ctype):
    block = np.arange(35.0).reshape(7, 5)
    st, kept = M.fill_container(block, ctype)
    assert st.size == 5
    for i, name in enumerate(ROWS):
        np.testing.assert_array_equal([getattr(st, name)[j] for j in range(5)], kept[i])


@pytest.mark.parametrize("ctype", [ctypes.c_float, ctypes.c_double])
def test_container_of_a_short_block_is_refused(ctype):
    """A missing row is an error, not a null pointer for the native code."""
    with pytest.raises(IndexError):
        M.fill_container(np.zeros((6, 5)), ctype)


@pytest.mark.parametrize("ctype", [ctypes.c_float, ctypes.c_double])
def test_container_takes_the_first_rows_of_a_taller_block(ctype):
    st, kept = M.fill_container(np.arange(60.0).reshape(12, 5), ctype)
    np.testing.assert_array_equal([st.area[j] for j in range(5)], kept[6])


def test_bundle_of_another_height_is_refused():
    for rows in (11, 13):
        with pytest.raises(AssertionError):
            M.bundle(S.c2Bundlef, np.zeros((rows, 4), np.float32), ctypes.c_float)

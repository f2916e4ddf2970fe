"""Rules of the search kernels over row numbers, on the host."""
import ctypes as C

import pytest

from hostlib import build_host


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    L = build_host("rows", tmp_path_factory.mktemp("host"))
    L.rows_text_mode.argtypes = [C.c_int32, C.c_uint32]
    return L


@pytest.mark.parametrize("jl", [0, 1, 0xdfffffff, 0xe0000000, 0xefffffff, 0xf0000000, 0xf0000001, 0xfffffffe])
def test_a_row_is_no_text_state(rows, jl):
    """A walker's neighbour interval may begin at any row of a text of up to
    2^32 - 2 bases.  Only an index with text mode, whose rows end below the
    marks, has walkers in it."""
    assert not rows.rows_text_mode(0, jl)
    assert rows.rows_text_mode(4, jl) == (jl >= 0xf0000000)

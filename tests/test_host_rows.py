"""Rules of the search kernels over row numbers, on the host."""
import ctypes as C

import pytest

from hostlib import build_host


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    L = build_host("rows", tmp_path_factory.mktemp("host"))
    L.rows_text_mode.argtypes = [C.c_int32, C.c_uint32]
    L.rows_clear_in_kernel.argtypes = [C.c_uint32, C.c_uint32, C.c_uint64]
    L.rows_put_walker.argtypes = [C.c_uint64, C.c_int32, C.POINTER(C.c_uint32 * 6)]
    return L


@pytest.mark.parametrize("jl", [0, 1, 0xdfffffff, 0xe0000000, 0xefffffff, 0xf0000000, 0xf0000001, 0xfffffffe])
def test_a_row_is_no_text_state(rows, jl):
    """A walker's neighbour interval may begin at any row of a text of up to
    2^32 - 2 bases.  Only an index with text mode, whose rows end below the
    marks, has walkers in it."""
    assert not rows.rows_text_mode(0, jl)
    assert rows.rows_text_mode(4, jl) == (jl >= 0xf0000000)


@pytest.mark.parametrize("length", [150, 2**30 - 1, 2**30, 2**31 - 1])
@pytest.mark.parametrize("entry", [0, 2, 3])
def test_a_reserved_entry_is_a_walker_or_a_hole(rows, entry, length):
    """The walk pass reads every entry a warp reserved: none may keep what an
    earlier pass left there, also where the read's anchors do not fit."""
    w = (C.c_uint32 * 6)()
    there = rows.rows_put_walker(entry, length, C.byref(w))
    assert there == (entry < 3 and length < 2**30)
    if there:
        assert list(w) == [7, 0x80000000 | 0x40000000 | 5, 1, 2, 3, 4]
    else:
        assert w[0] == (0xffffffff if entry < 3 else 0x55555555)


@pytest.mark.parametrize("reads", [1, 200, 256, 257, 10_000, 131_072])
def test_who_clears_the_record_mask(rows, reads):
    """The first kernel of a small batch does not clear the mask that a large
    one left: a thread has at most 64 words of it."""
    threads = 256 * min(-(-reads // 256), 4864)
    assert rows.rows_clear_in_kernel(reads, 256, 64 * threads)
    assert not rows.rows_clear_in_kernel(reads, 256, 64 * threads + 1)
    assert not rows.rows_clear_in_kernel(reads, 256, 10**9 // 32 * 64)

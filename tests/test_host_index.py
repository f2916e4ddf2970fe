"""The device memory that an index takes, on a fake CUDA runtime."""
import ctypes as C

import numpy as np
import pytest

from hostlib import build_host

MIB = 1 << 20
BASES = 8 * MIB
START, TWO_BASE = 1024 * MIB, 4 * BASES     # the start table of 13 bases; steps of two


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    L = build_host("index", tmp_path_factory.mktemp("host"))
    for f in ("fake_held", "fake_pinned_bytes"):
        getattr(L, f).restype = C.c_size_t
    L.fake_have.argtypes = [C.c_size_t]
    return L


@pytest.fixture
def index(host):
    h = C.c_void_p()
    L2 = np.array([BASES // 4 * i for i in (1, 2, 3, 4)], np.uint32)
    words = np.zeros(4 * (BASES // 64 + 1) + BASES // 16, np.uint32)
    samples = np.zeros((BASES + 7) // 7 - 1, np.uint32)
    p = [C.c_void_p(a.ctypes.data) for a in (L2, words, samples)]
    assert host.gs_index_from_host(5, p[0], p[1], C.c_uint64(words.size), 7, p[2], C.c_uint64(samples.size), 0,
                                   C.byref(h)) == 0
    yield h
    host.fake_have(0)
    host.gs_index_free(h)
    assert host.fake_held() == 0 and host.fake_errors() == 0


def _info(host, h):
    import gpuseed_gb300 as gs
    info = gs.IndexInfo()
    assert host.gs_index_get_info(h, C.byref(info)) == 0
    assert info.device_bytes == host.fake_held()
    return info


def test_least_memory(host, index):
    """set_kmer_len(13) gives back the start table and the two-base table; a
    longer one takes both again."""
    full = _info(host, index).device_bytes
    assert host.gs_index_set_kmer_len(index, 13) == 0
    info = _info(host, index)
    assert info.kmer_len == 13
    assert full - info.device_bytes == pytest.approx(START + TWO_BASE, abs=MIB)
    assert host.gs_index_set_kmer_len(index, 14) == 0
    info = _info(host, index)
    assert info.kmer_len == 14
    assert info.device_bytes - full == pytest.approx(3 * START, abs=MIB)


@pytest.mark.parametrize("room", [48, 52, 60, 64, 200])
def test_asked_for_comes_before_unasked(host, index, room):
    """The text structures (4 + 1/4 + 2 bytes a base, and one while they are
    made: 58 MiB) and a start table fit where they fit before loading made a
    two-base table (32 MiB) of its own accord."""
    full = _info(host, index).device_bytes
    assert host.gs_index_set_kmer_len(index, 14) == 0
    held = _info(host, index).device_bytes
    assert held > full
    host.fake_have(held - TWO_BASE + room * MIB)
    fits = room >= 59
    assert host.gs_index_set_text(index, 4) == (0 if fits else -4)
    info = _info(host, index)
    assert info.text_min == (4 if fits else 0)
    if not fits:
        assert info.device_bytes == held
    kept = room >= 59 + 32     # the two-base table: where both fit, or the text did not even without it
    if fits:
        assert info.device_bytes == pytest.approx(held + 6.25 * BASES - (0 if kept else TWO_BASE), abs=MIB)
    # a longer start table in the place of this one
    host.fake_have(info.device_bytes + 12 * START - (TWO_BASE if kept else 0))
    assert host.gs_index_set_kmer_len(index, 15) == 0
    assert _info(host, index).kmer_len == 15


def test_each_allocation_of_the_text_fails(host, index):
    """One allocation fails: the structures are made without the two-base
    table; when the next fails too, the call says so and frees all it took."""
    for at in range(1, 6):
        assert host.gs_index_set_kmer_len(index, 14) == 0
        held = _info(host, index).device_bytes
        host.fake_fail(at)
        assert host.gs_index_set_text(index, 4) == 0
        host.fake_fail(0)
        info = _info(host, index)
        assert info.device_bytes == pytest.approx(held + 6.25 * BASES - TWO_BASE, abs=MIB)
        assert host.gs_index_set_text(index, 0) == 0

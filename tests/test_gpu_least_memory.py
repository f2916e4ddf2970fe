"""An index in the least memory (set_kmer_len(13)): no start table, and walks
by one base, without the table for two.  As loaded, then without the tables,
then with a longer start table again; every record and position must be the
oracle's (integers: exact)."""
import pytest

from helpers import build_index, pack, random_reference
from test_gpu_start import _reads

pytestmark = pytest.mark.gpu


@pytest.fixture
def index(built, tmp_path):
    import gpuseed_gb300 as gs
    import pyoracle
    codes = random_reference(20_000, 31, dups=60)
    prefix = build_index(tmp_path, codes)
    return gs.Index(prefix), pyoracle.Index(prefix), pack(_reads(codes, 13, 7))


@pytest.mark.parametrize("text", [0, 1], ids=["walk", "text"])
def test_same_seeds(index, text):
    import gpuseed_gb300 as gs
    gidx, oidx, (seqs, offs, lens) = index
    gidx.set_text(text)
    ctx = gs.Context(gidx)
    held = []
    for kx in (None, 13, 15):
        if kx:
            gidx.set_kmer_len(kx)
        held.append(gidx.info().device_bytes)
        for slots in (0, 1):      # walks in the walk pass, and in the leftover pass
            for k in (13, 14, 16, 22):
                for n_mode in (0, 1):
                    for smem in (False, True):
                        got = ctx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode, walker_slots=slots)
                        want = oidx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode)
                        for r in range(lens.size):
                            assert got.read_records(r) == want.read_records(r), \
                                f"kx={kx} slots={slots} k={k} n_mode={n_mode} smem={smem} read {r}"
    ctx.close()
    assert held[1] < held[0] < held[2]

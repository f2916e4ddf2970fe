"""Output seeds merged by a warp per read (small batches, long reads) or by a
thread per read, on both sides of each line, against the oracle (integers:
exact)."""
import numpy as np
import pytest

from helpers import build_index, pack, random_reference, sample_reads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def index(built, tmp_path_factory):
    import gpuseed_gb300 as gs
    import pyoracle
    r = np.random.default_rng(3)
    unit = r.integers(0, 4, 400, dtype=np.uint8)
    parts = [random_reference(6000, 9)]
    for _ in range(40):   # diverged repeats: many records that begin or end alike
        u = unit.copy()
        at = r.integers(0, 400, 30)
        u[at] = r.integers(0, 4, 30)
        parts += [u, r.integers(0, 4, 20, dtype=np.uint8)]
    codes = np.concatenate(parts).astype(np.uint8)
    prefix = build_index(tmp_path_factory.mktemp("emit"), codes)
    return gs.Index(prefix), pyoracle.Index(prefix), codes


# 1 and 9 reads: a warp and a block; 4096 short reads are a warp's each, one
# more is a thread's; 16 items a read on average are a warp's in any number
@pytest.mark.parametrize("n,lengths", [(1, (4000,)), (9, (60, 150, 4000)), (4096, (40, 80, 150)),
                                       (4097, (40, 80, 150)), (4097, (490, 520)), (4200, (700, 1500))])
@pytest.mark.parametrize("kx", [13, 15])
def test_emit(index, n, lengths, kx):
    import gpuseed_gb300 as gs
    gidx, oidx, codes = index
    gidx.set_kmer_len(kx)
    ctx = gs.Context(gidx)
    try:
        some = sample_reads(codes, min(n, 40), seed=n, lengths=lengths, err=0.03, n_rate=0.1)
        seqs, offs, lens = pack([some[i % len(some)] for i in range(n)])
        oseqs, ooffs, olens = pack(some)
        for smem in (True, False):
            got = ctx.seed(seqs, offs, lens, k=18, smem=smem)
            want = oidx.seed(oseqs, ooffs, olens, k=18, smem=smem)
            records = [want.read_records(i) for i in range(len(some))]
            ns, npos = got.read_seed_off, got.read_pos_off
            for i in [*range(min(n, 80)), *range(n // 2, min(n, n // 2 + 40)), *range(max(0, n - 41), n)]:
                assert got.read_records(i) == records[i % len(some)], f"smem={smem} read {i}"
            # every read's counts are its copy's
            k = len(some)
            ds, dp = np.diff(ns.astype(np.int64)), np.diff(npos.astype(np.int64))
            idx = np.arange(n) % k
            assert (ds == ds[:k][idx]).all() and (dp == dp[:k][idx]).all()
    finally:
        ctx.close()
        gidx.set_kmer_len(13)

"""The batched start pass on its edges, against the oracle.

Its work items are 30 read windows, each window's two candidates settled
where they can be by the start table's entry: the one- and two-base left
extensions that an interval of at most 255 rows has.  The reads here end
windows at every place of an item, hold letters that the two strands' code
tables treat differently, start at odd addresses, lie at both ends of the
text and in repeats of 254 to 257 copies; every record and position must be
the oracle's (integers: exact).
"""
import random

import numpy as np
import pytest

from helpers import build_index, pack, sample_reads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def repeats(built, tmp_path_factory):
    import gpuseed_gb300 as gs
    import pyoracle

    r = np.random.default_rng(5)
    parts = [r.integers(0, 4, 4000, dtype=np.uint8)]
    for copies in (2, 3, 254, 255, 256, 257):
        unit = r.integers(0, 4, 45, dtype=np.uint8)
        for _ in range(copies):
            parts += [unit, r.integers(0, 4, int(r.integers(1, 9)), dtype=np.uint8)]
    parts += [r.integers(0, 4, 4001, dtype=np.uint8), np.zeros(40, np.uint8)]
    codes = np.concatenate(parts)
    prefix = build_index(tmp_path_factory.mktemp("start"), codes)
    return gs.Index(prefix), pyoracle.Index(prefix), codes


def _reads(codes, kx, seed):
    rng = random.Random(seed)
    text = "".join("ACGT"[c] for c in codes)
    lengths = sorted({kx, kx + 1, kx + 2, kx + 3, *range(kx + 28, kx + 33),
                      *range(kx + 58, kx + 63), 150, 301})
    reads = sample_reads(codes, 500, seed, lengths=lengths, err=0.02, n_rate=0.3)
    for n in lengths:
        reads += [text[:n].encode(), text[-n:].encode(), text[1:1 + n].encode()]
        for letter in "RUMB-EJ\rNacgtKSW":
            at = rng.randrange(0, len(text) - n)
            s = list(text[at:at + n])
            s[rng.randrange(n)] = letter
            reads.append("".join(s).encode())
    rng.shuffle(reads)
    return reads


@pytest.mark.parametrize("text", [0, 1], ids=["walk", "text"])
@pytest.mark.parametrize("kx", [13, 14, 15, 16])
def test_start_settles_what_the_walk_would(repeats, kx, text):
    import gpuseed_gb300 as gs

    gidx, oidx, codes = repeats
    gidx.set_kmer_len(kx)
    gidx.set_text(text)
    try:
        ctx = gs.Context(gidx)
        seqs, offs, lens = pack(_reads(codes, kx, 100 + kx))
        for k in (kx + 1, kx + 2, kx + 3, kx + 9):
            for n_mode in (0, 1):
                for smem in (False, True):
                    got = ctx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode)
                    want = oidx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode)
                    for r in range(lens.size):
                        assert got.read_records(r) == want.read_records(r), \
                            f"kx={kx} k={k} n_mode={n_mode} smem={smem} read {r}"
        ctx.close()
    finally:
        gidx.set_text(0)
        gidx.set_kmer_len(13)

"""Start table entries of one to three rows, which hold each row's six (or
three) bases before and the base after: against the oracle.

Units occur one to five times (four and five: the other entry form), with
copies that share 0 to 8 bases before them and are followed by the same base
or another; at both ends of the text too, where a row has fewer bases before
it or none after.  The reads take a copy with its surroundings and change one
base at each distance from the unit's ends; every record and position must be
the oracle's (integers: exact).
"""
import numpy as np
import pytest

from helpers import build_index, pack

pytestmark = pytest.mark.gpu

UNIT = 24


@pytest.fixture(scope="module")
def copies(built, tmp_path_factory):
    import gpuseed_gb300 as gs
    import pyoracle

    r = np.random.default_rng(11)
    rnd = lambda n: r.integers(0, 4, n, dtype=np.uint8)
    head, tail = rnd(UNIT), rnd(UNIT)
    parts, at, reads = [head], [], []
    total = UNIT
    for n in (1, 2, 3, 4, 5):
        for shared in range(9):
            for other in (False, True):
                unit, before, after = rnd(UNIT), rnd(shared), rnd(9)
                for c in range(n):
                    a = after.copy()
                    if other and c:
                        a[0] = (a[0] + c) % 4
                    # the base before the shared ones differs from copy to copy
                    block = np.concatenate([rnd(12), [np.uint8(c % 4)], before, unit, a]).astype(np.uint8)
                    at.append(total + 13 + shared)
                    parts.append(block)
                    total += block.size
    # the ends of the text, once more inside it
    parts += [rnd(20), head, rnd(20), tail, rnd(20), head, rnd(7), tail]
    codes = np.concatenate(parts).astype(np.uint8)
    at += [0, codes.size - UNIT, total + 20, total + 20 + UNIT + 20]
    for p in at:
        lo, hi = max(p - 14, 0), min(p + UNIT + 9, codes.size)
        s = codes[lo:hi]
        for q in [None, *range(lo, p), *range(p + UNIT, hi)][:: 1 if p < 4000 else 3]:
            t = s.copy()
            if q is not None:
                t[q - lo] ^= 1 + (p % 3)
            reads.append("".join("ACGT"[c] for c in (t if p % 2 else 3 - t[::-1])).encode())
    prefix = build_index(tmp_path_factory.mktemp("rows"), codes)
    return gs.Index(prefix), pyoracle.Index(prefix), pack(reads)


@pytest.mark.parametrize("text", [0, 1], ids=["walk", "text"])
@pytest.mark.parametrize("kx", [13, 14, 15, 16])
def test_few_rows(copies, kx, text):
    import gpuseed_gb300 as gs

    gidx, oidx, (seqs, offs, lens) = copies
    gidx.set_kmer_len(kx)
    gidx.set_text(text)
    ctx = gs.Context(gidx)
    try:
        for k in (kx + 1, kx + 4, kx + 7):
            for smem in (False, True):
                got = ctx.seed(seqs, offs, lens, k=k, smem=smem)
                want = oidx.seed(seqs, offs, lens, k=k, smem=smem)
                for r in range(lens.size):
                    assert got.read_records(r) == want.read_records(r), f"kx={kx} k={k} smem={smem} read {r}"
    finally:
        ctx.close()
        gidx.set_text(0)
        gidx.set_kmer_len(13)

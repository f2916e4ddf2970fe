"""Walks by two bases a step, against the oracle (integers: exact): texts that
end about the 64-row blocks, of repeats whose walks keep several rows, and
reads that end, hold an odd letter or differ at every distance from their
start strings, so that a walk's last step is by one base or two, with and
without its neighbour's interval."""
import random

import numpy as np
import pytest

from helpers import build_index, pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,period", [(62, 1), (63, 5), (64, 3), (65, 2), (126, 31), (127, 20), (128, 31),
                                      (129, 16), (700, 45), (3000, 61)])
def test_two_base_steps(built, tmp_path, n, period):
    import gpuseed_gb300 as gs
    import pyoracle
    r = np.random.default_rng(n)
    codes = np.resize(r.integers(0, 4, period, dtype=np.uint8), n).astype(np.uint8)
    at = r.integers(0, n, max(1, n // 60))
    codes[at] = r.integers(0, 4, at.size)
    prefix = build_index(tmp_path, codes)
    gidx, oidx = gs.Index(prefix), pyoracle.Index(prefix)
    text = "".join("ACGT"[c] for c in codes)
    comp = str.maketrans("ACGT", "TGCA")
    rng = random.Random(n)
    reads = [text.encode(), text.translate(comp)[::-1].encode()]
    for i in range(600):
        length = rng.randrange(15, min(n, 90) + 1)
        s = rng.randrange(0, n - length + 1)
        t = list(text[s:s + length])
        for _ in range(i % 3):
            t[rng.randrange(length)] = rng.choice("ACGTACGTNRX")
        t = "".join(t)
        reads.append((t if i % 2 else t.translate(comp)[::-1]).encode())
    seqs, offs, lens = pack(reads)
    ctx = gs.Context(gidx)
    for k in (14, 15, 18):
        for n_mode in (0, 1):
            for smem in (False, True):
                got = ctx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode)
                want = oidx.seed(seqs, offs, lens, k=k, smem=smem, n_mode=n_mode)
                for i in range(lens.size):
                    assert got.read_records(i) == want.read_records(i), f"k={k} n_mode={n_mode} smem={smem} {i}"
    ctx.close()

"""Positions by LF chains, with and without tiles of more than one round of 32
(a batch of more than 311,296 positions), against the oracle: every sampling
distance, repeats whose seeds spread over many tiles, a last round that is
not whole (integers: exact)."""
import numpy as np
import pytest

from helpers import build_index, pack, sample_reads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("intv", [1, 2, 7, 64])
@pytest.mark.parametrize("reads", [37, 8001])
def test_positions(built, tmp_path, intv, reads):
    import gpuseed_gb300 as gs
    import pyoracle
    r = np.random.default_rng(intv)
    unit = r.integers(0, 4, 120, dtype=np.uint8)
    parts = [r.integers(0, 4, 500, dtype=np.uint8)]
    for _ in range(130):
        u = unit.copy()
        u[r.integers(0, 120)] = r.integers(0, 4)
        parts += [u, r.integers(0, 4, int(r.integers(0, 5)), dtype=np.uint8)]
    codes = np.concatenate(parts).astype(np.uint8)
    prefix = build_index(tmp_path, codes, sa_intv=intv)
    some = sample_reads(codes[500:], 40, seed=intv, lengths=(30, 60, 110))
    seqs, offs, lens = pack([some[i % 40] for i in range(reads)])
    oseqs, ooffs, olens = pack(some)
    oidx = pyoracle.Index(prefix)
    ctx = gs.Context(gs.Index(prefix))
    for lf_mode in (0, 1):
        got = ctx.seed(seqs, offs, lens, k=20, smem=False, lf_mode=lf_mode)
        want = oidx.seed(oseqs, ooffs, olens, k=20, smem=False, lf_mode=lf_mode)
        assert reads < 8000 or got.pos.size > 152 * 8 * 8 * 32
        records = [want.read_records(i) for i in range(40)]
        for i in range(reads):
            assert got.read_records(i) == records[i % 40], f"lf_mode={lf_mode} read {i}"
    ctx.close()

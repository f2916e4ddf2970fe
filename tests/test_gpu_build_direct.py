"""The builder's device-to-device route: an index built without files is the
index that its files load, and a code that is no base is named."""
import os

import numpy as np
import pytest

from helpers import pack, random_reference, sample_reads

pytestmark = pytest.mark.gpu


def _text(n, period):
    return random_reference(n, n) if not period else np.resize(random_reference(period, n), n).astype(np.uint8)


# ends of a 64-row block, the smallest texts, and texts whose suffixes stay
# unresolved for many rounds (a period of 1, 2 and 333 bases)
@pytest.mark.parametrize("n,period,intv", [(1, 0, 1), (2, 0, 7), (63, 0, 7), (64, 0, 1), (65, 0, 64), (128, 0, 3),
                                           (4097, 0, 7), (3000, 1, 7), (5001, 2, 5), (20_000, 333, 7),
                                           (100_000, 0, 7)])
def test_built_index_is_the_loaded_one(built, tmp_path, n, period, intv):
    import gpuseed_gb300 as gs
    import pyoracle
    codes = _text(n, period)
    prefix = os.path.join(str(tmp_path), "o")
    pyoracle.build_index(codes, intv, prefix)
    a, b = gs.build_index(codes, intv), gs.Index(prefix)
    assert bytes(a.info()) == bytes(b.info())
    lengths = [v for v in (14, 20, 50, 150) if v <= n]
    if not lengths:
        return
    seqs, offs, lens = pack(sample_reads(codes, 60, seed=n, lengths=tuple(lengths)))
    x, y = (gs.Context(i).seed(seqs, offs, lens, k=14, smem=False) for i in (a, b))
    assert (x.read_seed_off == y.read_seed_off).all() and (x.read_pos_off == y.read_pos_off).all()
    assert (x.seeds == y.seeds).all() and (x.pos == y.pos).all()


@pytest.mark.parametrize("n,at", [(1, 0), (257, 0), (257, 256), (100_000, 77_777)])
def test_code_out_of_range_is_named(built, n, at):
    import gpuseed_gb300 as gs
    codes = random_reference(n, 2)
    codes[at:] = 4 + (np.arange(n - at) % 200).astype(np.uint8)
    with pytest.raises(gs.GsError, match=f"code 4 at {at} is not 0..3"):
        gs.build_index(codes, 7)

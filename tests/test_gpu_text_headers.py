"""Headers of the text records, a warp per read: batches about a block's
eight reads and past one round of the device's blocks, number widths that
change within a warp's reads, against the host writer (bytes: exact)."""
import numpy as np
import pytest

from helpers import build_index, pack, random_reference, sample_reads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def index(built, tmp_path_factory):
    import gpuseed_gb300 as gs
    codes = random_reference(3000, 4)
    return gs.Index(build_index(tmp_path_factory.mktemp("headers"), codes)), codes


@pytest.mark.parametrize("n,first", [(1, 0), (1, 9), (7, 4), (8, 95), (9, 996), (33, 99_999_980),
                                     (40_000, 4_294_950_000)])
def test_headers(index, tmp_path, n, first):
    import gpuseed_gb300 as gs
    idx, codes = index
    some = sample_reads(codes, min(n, 50), seed=n, lengths=(10, 25, 40))
    seqs, offs, lens = pack([some[i % len(some)] for i in range(n)])
    ctx = gs.Context(idx)
    for smem in (False, True):
        ctx.seed(seqs, offs, lens, k=19, smem=smem)
        out = []
        for host in (False, True):
            p = tmp_path / f"{smem}{host}"
            with open(p, "wb") as f:
                ctx.write_text(f.fileno(), first, smem, host=host)
            out.append(np.frombuffer(p.read_bytes(), np.uint8))
        assert out[0].size == out[1].size and (out[0] == out[1]).all()
    ctx.close()

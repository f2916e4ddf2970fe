"""The per-read offsets and the position -> seed map at the sizes where their
blocks, tiles and rounds end, against the oracle.

Offsets of slots, work items, seeds and positions come from sums of blocks of
256 reads and scans within them; positions are resolved in rounds of 32 and
tiles of up to 256.  Batches of 1, 255, 256, 257 and 4,000 reads put the ends
everywhere, with reads too short for a seed among them, and a unit of 700
copies gives seeds whose positions span many tiles (integers: exact).
"""
import numpy as np
import pytest

from helpers import build_index, pack, sample_reads

pytestmark = pytest.mark.gpu


def text_of(codes):
    return "".join("ACGT"[c] for c in codes)


@pytest.fixture(scope="module")
def copies(built, tmp_path_factory):
    import gpuseed_gb300 as gs
    import pyoracle

    r = np.random.default_rng(11)
    unit = r.integers(0, 4, 60, dtype=np.uint8)
    parts = [r.integers(0, 4, 9000, dtype=np.uint8)]
    for _ in range(700):
        parts += [unit, r.integers(0, 4, int(r.integers(1, 6)), dtype=np.uint8)]
    codes = np.concatenate(parts)
    prefix = build_index(tmp_path_factory.mktemp("offsets"), codes)
    reads = sample_reads(codes, 4000, 12, lengths=(10, 19, 20, 40, 80, 150), err=0.01, n_rate=0.1)
    return gs.Index(prefix), pyoracle.Index(prefix), reads, codes


@pytest.mark.parametrize("text", [0, 4], ids=["lf_walk", "full_sa"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 4000])
def test_offsets_and_positions(copies, n, text):
    import torch

    import gpuseed_gb300 as gs

    gidx, oidx, reads, _ = copies
    gidx.set_text(text)
    seqs, offs, lens = pack(reads[-n:])
    dev = [torch.from_numpy(np.frombuffer(seqs, np.uint8).copy()).cuda(),
           torch.from_numpy(offs.view(np.int64)).cuda(), torch.from_numpy(lens.view(np.int32)).cuda()]
    ctx = gs.Context(gidx)
    for smem in (True, False):
        want = oidx.seed(seqs, offs, lens, k=19, smem=smem)
        torch.cuda.synchronize()
        # the first pass of a context, a repeated one, and a captured one twice
        for graph in (False, False, True, True):
            got = ctx.seed_device(*(t.data_ptr() for t in dev), n, fetch=True, k=19, smem=smem,
                                  graph=graph)
            assert got.read_seed_off[-1] == got.seeds.shape[0]
            assert got.read_pos_off[-1] == got.pos.size
            for r in range(n):
                assert got.read_records(r) == want.read_records(r), f"n={n} smem={smem} read {r}"
    ctx.close()
    gidx.set_text(0)


def test_batches_of_any_size_through_one_context(copies):
    """A context runs small batches in one go on the room and the sizes of
    the passes before: reads with far more slots, seeds or positions than
    those expected make it run again, with the same result."""
    import torch

    import gpuseed_gb300 as gs

    gidx, oidx, reads, codes = copies
    full = [r for r in reads if len(r) == 150]
    # inside the repeated unit: one seed of 700 positions
    unit = text_of(codes)[9005:9055].encode()
    batches = [reads[:1], [b"ACGT"] * 40, reads[:700], full * 3, [unit] * 300, reads[5:9], reads * 3]
    ctx = gs.Context(gidx)
    for i, batch in enumerate(batches):
        seqs, offs, lens = pack(batch)
        want = oidx.seed(seqs, offs, lens, k=19, smem=True)
        d = [torch.from_numpy(np.frombuffer(seqs, np.uint8).copy()).cuda(),
             torch.from_numpy(offs.view(np.int64)).cuda(), torch.from_numpy(lens.view(np.int32)).cuda()]
        torch.cuda.synchronize()
        results = [ctx.seed(seqs, offs, lens, k=19, smem=True)]
        for graph in (False, True, False, True):
            results.append(ctx.seed_device(*(t.data_ptr() for t in d), lens.size, fetch=True, k=19,
                                           smem=True, graph=graph))
        for j, got in enumerate(results):
            for r in range(lens.size):
                assert got.read_records(r) == want.read_records(r), f"batch {i} call {j} read {r}"
    ctx.close()

"""The seeding context's host code on a fake CUDA runtime: what a pass is
sized by, and what a failed one leaves behind."""
import ctypes as C

import numpy as np
import pytest

from hostlib import build_host

ENOMEM = -4


class Pass(C.Structure):
    _fields_ = [(n, C.c_uint64) for n in ("passes", "n_items", "item_cap", "item_read_cap", "slot_cap",
                                          "walker_cap", "clear_words", "mask_words", "items", "slots",
                                          "seeds_a_read", "pos_a_read")]


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    L = build_host("pass", tmp_path_factory.mktemp("host"))
    L.fake_pass.restype = C.POINTER(Pass)
    L.fake_index.restype = C.c_void_p
    L.fake_pinned_bytes.restype = C.c_size_t
    return L


class Seeder:
    """A context, and passes over reads of given lengths"""

    def __init__(self, L):
        self.L, self.h = L, C.c_void_p()
        assert L.gs_ctx_create(C.c_void_p(L.fake_index()), None, C.byref(self.h)) == 0
        p = L.fake_pass().contents
        p.seeds_a_read, p.pos_a_read = 2, 3

    def run(self, lengths, device=True, fetch=0, **kw):
        import gpuseed_gb300 as gs
        p = gs.Context.params(**dict({"k": 19, "smem": True}, **kw))
        lens = np.asarray(lengths, np.uint32)
        self.offs = np.zeros(lens.size, np.uint64)
        self.offs[1:] = np.cumsum(lens[:-1], dtype=np.uint64)
        self.lens, self.seqs = lens, np.zeros(int(lens.sum(dtype=np.uint64)) + 1, np.uint8)
        a = [C.c_void_p(v.ctypes.data) for v in (self.seqs, self.offs, self.lens)]
        if device:
            rc = self.L.gs_seed_device(self.h, *a, lens.size, C.byref(p), fetch)
        else:
            rc = self.L.gs_seed(self.h, *a, lens.size, C.byref(p))
        assert self.L.fake_errors() == 0
        return rc

    @property
    def last(self):
        return self.L.fake_pass().contents

    def close(self):
        self.L.gs_ctx_free(self.h)


@pytest.fixture
def seeder(host):
    s = Seeder(host)
    yield s
    host.fake_fail(0)
    s.close()


def test_record_mask_of_a_pass_that_had_no_memory(seeder):
    """Each allocation of a pass larger than the one before fails in turn; the
    batch then runs in parts, on the same context.  No pass clears or marks
    more of the record mask than there is (the slots may have been had, and
    the mask not)."""
    assert seeder.run([100] * 2000) == 0
    for at in range(1, 40):
        seeder.L.fake_fail(at)
        rc = seeder.run([100 + at] * (2000 + 600 * at))
        seeder.L.fake_fail(0)
        assert rc in (0, ENOMEM)
        for _ in range(2):
            assert seeder.run([100] * 1500) == 0
            assert (seeder.last.slot_cap + 31) // 32 <= seeder.last.mask_words


def test_captured_pass_of_smaller_buffers(seeder):
    """A captured pass stops at the sizes it was captured with: it is not
    replayed where a buffer is larger since, although it lies where it lay."""
    assert seeder.run([100] * 2000, graph=1) == 0
    answers = []
    for which in range(20):
        answers.append(seeder.L.fake_replayed_when_larger(seeder.h, which))
        if answers[-1] < 0:
            break
    assert answers == [0] * 9 + [-1]


def test_a_pass_is_sized_for_its_batch(seeder):
    """Batches of any size after one another: the pass whose result is taken
    was sized for the batch's work items, slots and walkers, whatever the
    batches before it had, and a full walker buffer that was sized for fewer
    items is no reason for a larger one."""
    rng = np.random.default_rng(1)
    batches = [[100] * 3000, [12] * 500, [100] * 3000, [150] * 40, [9000], [150] * 100, [30] * 3000, [250] * 3000]
    batches += [[int(np.exp(rng.uniform(2.3, 7)))] * int(np.exp(rng.uniform(0, 8))) for _ in range(60)]
    for batch in batches:
        assert seeder.run(batch) == 0
        p = seeder.last
        assert p.items <= p.item_cap and p.slots <= p.slot_cap, batch[:1]
        assert p.items * 16 < p.walker_cap, batch[:1]


def test_alike_batches_run_once(seeder):
    """Batches of one kind, or of two that take turns, are searched once each
    from the second on."""
    for kinds in ([100], [100, 150], [100, 10]):
        for i in range(8):
            before = seeder.last.passes
            assert seeder.run([kinds[i % len(kinds)]] * 3000) == 0
            assert i < 2 or seeder.last.passes == before + 1, f"{kinds} {i}"
            assert i < 2 or seeder.last.clear_words, "in one go"


@pytest.mark.parametrize("device", [True, False])
@pytest.mark.parametrize("before", [[(10_000, 2)], [(10_000, 1)], [(9000, 0)], [(9000, 0), (10_000, 2), (10_000, 0)]])
def test_other_batches_do_not_keep_one_from_running_once(host, device, before):
    """After passes (reads, kernel) of a smaller batch, whose room holds this
    one, and of the other kernels, which count work items otherwise."""
    s = Seeder(host)
    for n, kernel in before:
        assert s.run([100] * n, kernel=kernel) == 0
    for i in range(3):
        passes = s.last.passes
        assert s.run([100] * 10_000, device=device) == 0
        assert s.last.passes == passes + 1
        assert i < 1 or s.last.clear_words, "in one go"
    s.close()


def _timing(s):
    t = C.c_float(), C.c_float()
    assert s.L.gs_ctx_last_timing(s.h, C.byref(t[0]), C.byref(t[1])) == 0
    return t[0].value, t[1].value


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("ask", [False, True], ids=["later", "before"])
def test_timing_after_a_failed_pass(host, ask, graph):
    """The times are of the last pass that ended, also when they are asked for
    after one that failed on the way (each allocation in turn)."""
    for at in range(1, 30):
        s = Seeder(host)
        assert s.run([100] * 2000, graph=graph) == 0
        assert s.run([100] * 2000, graph=graph) == 0
        want = _timing(s) if ask else None
        host.fake_fail(at)
        rc = s.run([120] * 4000, graph=graph)
        host.fake_fail(0)
        search, total = _timing(s)
        assert 0 < search <= total
        if rc and ask:
            assert (search, total) == want
        s.close()


@pytest.mark.parametrize("reads", [300, 3000, 60_000])
def test_results_take_pinned_memory_once(host, reads):
    """A context that seeds batches of one kind from host buffers takes the
    memory it pins in its first pass, and no more than a first guess or a
    quarter above its results and its input."""
    s = Seeder(host)
    before = host.fake_pinned_bytes()
    taken = []
    for _ in range(4):
        assert s.run([100] * reads, device=False) == 0
        taken.append(host.fake_pinned_bytes() - before)
    assert taken[0] == taken[3]
    result = reads * (16 + 2 * 32 + 3 * 4)
    if reads > 4096:
        assert taken[0] < 1.3 * result
    s.close()


def test_served_requests_are_pinned_once(host):
    """A server's worker pins a merged batch's reads once, not once more for
    the pass to take them from."""
    import gpuseed_gb300 as gs
    p = host.fake_pass().contents
    p.seeds_a_read = p.pos_a_read = 0
    opts = gs.ServerOpts(1, 0, 0, gs.Context.params(k=19, smem=True))
    srv, rid = C.c_void_p(), C.c_uint64()
    before = host.fake_pinned_bytes()
    assert host.gs_server_start(C.c_void_p(host.fake_index()), C.byref(opts), C.byref(srv)) == 0
    n, length = 1000, 200
    lens = np.full(n, length, np.uint32)
    offs = np.arange(n, dtype=np.uint64) * length
    seqs = np.zeros(n * length, np.uint8)
    a = [C.c_void_p(v.ctypes.data) for v in (seqs, offs, lens)]
    assert host.gs_server_submit(srv, *a, n, C.byref(rid)) == 0
    assert host.gs_server_wait(srv, rid, -1) == 0
    host.gs_server_stop(srv)
    # with the offsets and lengths, and half as much again for the next; the
    # results' room: two offsets a read, and a guess at seeds and positions
    results = 1.25 * (n * 16 + (4 * n + 512) * 32 + (8 * n + 8192) * 4)
    assert host.fake_pinned_bytes() - before < 1.5 * n * (length + 12) + results + 16384

"""The work a user of gpuseed_gb300 has it do, as cases that can be timed.

A case names a genome (three sizes, each with the start table and the
structures its users would have), a batch of reads and the entry point that
takes them.  The genome's index is resident, as in any program that seeds
more than one batch: it is built once per process and shared.  Reads come
from the seed alone; every state has a context (or server) of its own.  The
program takes each pass's results into arrays of its own, sized once by the
batch (rows past a pass's results are zero).
"""
import ctypes
import functools
import math

import numpy as np
import torch

import gpuseed_gb300 as gs
from gpuseed_gb300 import workloads as W

# Genome sizes: a bacterial one (start table of 13 bases), a chromosome
# (14 bases) as loaded by default, and a human-sized one (16 bases) with the
# text structures that a long-running user builds.
GENOMES = {"bacterial": (1, 1_000_000, 0), "chromosome": (2, 100_000_000, 0),
           "human": (3, 3_100_000_000, 4)}

SHORT = "50,75,100,150,250"    # mixed short reads
LONG = "lognormal"             # median 2 kbp, 0.5 to 10 kbp


def case(name, kind, genome, reads, lengths, *, smem, k, sub=0.01, indel=0.0005, nrun=0.0,
         stop=False, bwa=False, max_occ=0, in_place=(0.0, 0.0)):
    """in_place: seeds and positions a read that the program of a host batch
    reads where the library left them; it copies those beyond"""
    c = {"kind": kind, "genome": genome, "reads": reads, "lengths": lengths, "smem": smem, "k": k,
         "sub": sub, "indel": indel, "nrun": nrun, "stop": stop, "bwa": bwa, "max_occ": max_occ,
         "seeds_in_place": in_place[0], "pos_in_place": in_place[1]}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one read looked up interactively: the latency of a call
        case("one_read", "host", "human", 1, "150", smem=True, k=19),
        # a client's request of a few hundred reads, host buffers in and out
        case("request", "host", "human", 300, "100-250", smem=True, k=19, indel=0.0),
        # a sequencing run of a small genome, batch after batch through the
        # same device buffers: a captured pass replayed
        case("bacterial_graph", "graph", "bacterial", 10_000, "100", smem=False, k=20, sub=0.005,
             indel=0.0),
        # a million 150-base reads on a chromosome, resident on the device,
        # the index as it is loaded by default
        case("chromosome_device", "device", "chromosome", 1_000_000, "150", smem=True, k=19,
             nrun=0.001),
        # the MEM mode from host buffers through the C entry points
        case("chromosome_mem_host", "host_c", "chromosome", 150_001, "150", smem=False, k=19,
             nrun=0.001, in_place=(2.4, 8.5)),
        # the bulk of the use: mixed short reads on a human-sized genome
        case("human_device", "device", "human", 2_000_000, SHORT, smem=True, k=19),
        # the same from pinned host buffers, a batch large enough to run in
        # chunks whose copies overlap the passes
        case("human_host", "host_c", "human", 4_300_000, SHORT, smem=True, k=19,
             in_place=(3.6, 4.35)),
        # long reads with many indels, MEM mode
        case("human_long", "device", "human", 40_000, LONG, smem=False, k=20, sub=0.02, indel=0.01),
        # the printed records (the command line's -o), formatted on the device
        case("text_records", "text", "chromosome", 100_000, "150", smem=False, k=20, nrun=0.001),
        # ragged very short reads, some shorter than k, with bwa's semantics
        # (N stops a match, bwa's LF) and a cap on occurrences
        case("strict_short", "device", "human", 60_007, "20-76", smem=True, k=25, sub=0.02,
             indel=0.0, nrun=0.01, stop=True, bwa=True, max_occ=500),
        # a burst of requests of 1 to 4096 reads on the serving loop
        case("serve_burst", "serve", "human", 16, "100-250", smem=True, k=19, indel=0.0),
        # a new genome: its index built, loaded, and a first batch seeded
        # (reads: of that batch; 10 Mbp)
        dict(case("index_build", "build", "new", 1_000, "150", smem=True, k=19), bases=10_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean(lengths):
    """The mean read length"""
    if lengths == LONG:
        return 2400
    each = [int(v) for v in lengths.replace("-", ",").split(",")]
    return sum(each) / len(each)


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "host", "host_c", "graph", "text",
                       "serve", "build"])
    if kind == "build":
        c = case(None, "build", "new", _log(rng, 1, 5_000), "150", smem=rng.random() < 0.5,
                 k=rng.randrange(15, 32))
        return dict(c, bases=_log(rng, 100_000, 12_000_000))
    genome = rng.choice(["bacterial", "chromosome", "human", "human"])
    lengths = rng.choice(["100", "150", SHORT, "100-250", "20-76", "31-301", LONG])
    mean = _mean(lengths)
    # up to 200 million bases; the text and the host copies of a batch less
    most = {"device": 200e6, "host": 2e6, "host_c": 50e6, "graph": 50e6, "text": 20e6}
    if kind == "serve":
        reads = rng.randrange(2, 17)
        lengths = rng.choice(["100-250", "100", "31-301"])
    else:
        reads = _log(rng, 1, max(2, most[kind] / mean))
    smem = rng.random() < 0.6
    if not smem and genome != "bacterial":
        reads = max(1, reads // 4)     # every match of a repeat is located
    low = {"bacterial": 13, "chromosome": 15, "human": 17}[genome] + (0 if smem else 2)
    return case(None, kind, genome, reads, lengths, smem=smem, k=rng.randrange(low, 34),
                sub=rng.choice([0.002, 0.01, 0.02, 0.05]), indel=rng.choice([0.0, 0.0005, 0.01]),
                nrun=rng.choice([0.0, 0.0, 0.01]), stop=rng.random() < 0.25,
                bwa=rng.random() < 0.25, max_occ=rng.choice([0, 0, 0, 50, 500]))


@functools.lru_cache(maxsize=None)
def _genome(name):
    """(index, codes, N mask) of a resident genome: at most the three above"""
    config, bases, text = GENOMES[name]
    codes, nmask = W.make_reference(W.ref_spec(config, bases))
    index = gs.build_index(codes, sa_intv=7)
    if text:
        index.set_text(text)
    return index, codes, nmask


def _reads(c, codes, nmask, seed, n):
    r = W.ReadSpec()
    r.seed, r.n_reads = 0x9E3779B97F4A7C15 * (seed + 1) & (2 ** 64 - 1), n
    r.sub_rate, r.indel_rate, r.indel_max = c["sub"], c["indel"], 3
    r.nrun_frac, r.nrun_min, r.nrun_max = c["nrun"], 1, 20
    if c["lengths"] == LONG:
        r.len_mode, r.ln_median, r.ln_sigma = W.LEN_LOGNORMAL, 2000.0, 0.6
        r.len_min, r.len_max = 500, 10000
    elif "," in c["lengths"]:
        each = [int(v) for v in c["lengths"].split(",")]
        r.len_mode, r.n_choices = W.LEN_CHOICE, len(each)
        for i, v in enumerate(each):
            r.len_choices[i] = v
    elif "-" in c["lengths"]:
        r.len_mode = W.LEN_UNIFORM
        r.len_min, r.len_max = (int(v) for v in c["lengths"].split("-"))
    else:
        r.len_mode, r.len_fixed = W.LEN_FIXED, int(c["lengths"])
    return W.make_reads(codes, nmask, r)


def _sizes(c):
    """The reads of each request of a burst, spread over 1 to 4096"""
    sizes = np.exp(np.random.default_rng(c["reads"]).uniform(0, math.log(4096), c["reads"]))
    return sizes.astype(np.int64).clip(1, 4096)


def _rows(reads, lengths):
    """Room for the seeds and positions of a batch"""
    bases = reads * _mean(lengths)
    return {"seeds": 1024 + int(0.1 * bases), "pos": 16384 + int(0.4 * bases)}


def _params(c):
    return {"k": c["k"], "smem": c["smem"], "n_mode": gs.N_STOP if c["stop"] else gs.N_WILDCARD,
            "lf_mode": gs.LF_BWA if c["bwa"] else gs.LF_GPUSEED, "max_occ": c["max_occ"]}


def prepare(c, seed):
    s = {"kind": c["kind"], "params": _params(c), "own": {}}
    if c["kind"] == "build":
        spec = W.ref_spec(2, c["bases"])
        spec.seed += 7919 * (seed + 1)
        s["codes"], nmask = W.make_reference(spec)
        s["reads"] = _reads(c, s["codes"], nmask, seed, c["reads"])
        s["room"] = _rows(c["reads"], c["lengths"])
        return s
    index, codes, nmask = _genome(c["genome"])
    if c["kind"] == "serve":
        sizes = _sizes(c)
        seqs, offs, lens = _reads(c, codes, nmask, seed, int(sizes.sum()))
        ends = np.cumsum(sizes)
        s["requests"] = [(seqs, offs[e - n:e].copy(), lens[e - n:e].copy())
                         for e, n in zip(ends, sizes)]
        s["room"] = [_rows(int(n), c["lengths"]) for n in sizes]
        s["own"] = [{} for _ in sizes]
        s["server"] = gs.Server(index, **s["params"])
        return s
    seqs, offs, lens = _reads(c, codes, nmask, seed, c["reads"])
    s["room"] = _rows(c["reads"], c["lengths"])
    t = [torch.from_numpy(v) for v in (seqs, offs.view(np.int64), lens.view(np.int32))]
    if c["kind"] in ("device", "graph", "text"):
        s["stream"] = torch.cuda.Stream()
        s["context"] = gs.Context(index, stream=s["stream"].cuda_stream)
        s["on_device"] = [v.cuda() for v in t]
        if c["kind"] == "text":
            # a header of about 160 bytes a read, 28 a seed, 12 a position
            s["room"] = {"text": 65536 + c["reads"] * 200 + 28 * s["room"]["seeds"]}
        like = {"seeds": ((8,), torch.int32), "pos": ((), torch.int32), "text": ((), torch.uint8)}
        for name, n in s["room"].items():
            s["own"][name] = torch.zeros((n, *like[name][0]), dtype=like[name][1], device="cuda")
        return s
    s["context"] = gs.Context(index)
    if c["kind"] == "host_c":
        s["pinned"] = [v.pin_memory() for v in t]
        s["in_place"] = {"seeds": int(c["seeds_in_place"] * c["reads"]),
                         "pos": int(c["pos_in_place"] * c["reads"])}
    else:
        s["reads"] = (seqs, offs, lens)
    return s


def _kept(own, name, rows, v):
    """`v` in the program's own array `name` of `rows` rows (as many doublings
    of that as it needs)"""
    while rows < v.shape[0]:
        rows *= 2
    if name not in own or own[name].shape[0] < rows:
        if isinstance(v, np.ndarray):
            own[name] = np.zeros((rows, *v.shape[1:]), v.dtype)
        else:
            own[name] = torch.zeros((rows, *v.shape[1:]), dtype=v.dtype, device=v.device)
    if isinstance(v, np.ndarray):
        own[name][:v.shape[0]] = v
    else:
        own[name][:v.shape[0]].copy_(v, non_blocking=True)
    return own[name]


class _Owned:
    """Memory that a context owns, as an array that keeps the context alive"""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.desc = {"data": (ctypes.cast(pointer, ctypes.c_void_p).value, False),
                     "shape": shape, "typestr": typestr, "version": 3}


class _OnDevice(_Owned):
    @property
    def __cuda_array_interface__(self):
        return dict(self.desc, version=2)


class _OnHost(_Owned):
    @property
    def __array_interface__(self):
        return self.desc


def _device_view(owner, pointer, shape, typestr, dtype):
    if not math.prod(shape):
        return torch.empty(shape, dtype=dtype, device="cuda")
    return torch.as_tensor(_OnDevice(owner, pointer, shape, typestr), device="cuda")


def _host_view(owner, pointer, shape, typestr):
    if not math.prod(shape):
        return np.zeros(shape, typestr)
    return np.asarray(_OnHost(owner, pointer, shape, typestr))


def _device_result(s):
    ctx, v = s["context"], gs.ResultView()
    gs.check(gs.lib().gs_result_device(ctx.h, ctypes.byref(v)))
    n, ns, npos = int(v.n_reads), int(v.n_seeds), int(v.n_pos)
    seeds = _device_view(ctx, v.seeds, (ns, 8), "<i4", torch.int32)
    pos = _device_view(ctx, v.pos, (npos,), "<i4", torch.int32)
    return {"seeds": _kept(s["own"], "seeds", s["room"]["seeds"], seeds),
            "pos": _kept(s["own"], "pos", s["room"]["pos"], pos),
            "read_seed_off": _device_view(ctx, v.read_seed_off, (n + 1,), "<i8", torch.int64),
            "read_pos_off": _device_view(ctx, v.read_pos_off, (n + 1,), "<i8", torch.int64)}


def _host_result(s):
    """The context's host arrays as a C caller reads them: in place up to the
    rows every batch of this kind has, the rest taken over"""
    ctx, v = s["context"], gs.ResultView()
    gs.check(gs.lib().gs_result_host(ctx.h, ctypes.byref(v)))
    n, ns, npos = int(v.n_reads), int(v.n_seeds), int(v.n_pos)
    out = {"read_seed_off": _host_view(ctx, v.read_seed_off, (n + 1,), "<i8"),
           "read_pos_off": _host_view(ctx, v.read_pos_off, (n + 1,), "<i8")}
    for name, p, shape in (("seeds", v.seeds, (ns, 8)), ("pos", v.pos, (npos,))):
        a, at = _host_view(ctx, p, shape, "<i4"), s["in_place"][name]
        out[name] = a[:at]
        room = 4096 + s["room"][name] // (16 if at else 1)
        out[name + "_rest"] = _kept(s["own"], name, room, a[at:])
    return out


def _of_result(r, own, room):
    return {"seeds": _kept(own, "seeds", room["seeds"], r.seeds.view(np.int32)),
            "pos": _kept(own, "pos", room["pos"], r.pos.view(np.int32)),
            "read_seed_off": r.read_seed_off.view(np.int64)}


def run(s):
    kind, params = s["kind"], s["params"]
    if kind == "host":
        r = s["context"].seed(*s["reads"], **params)
        return dict(_of_result(r, s["own"], s["room"]), read_pos_off=r.read_pos_off.view(np.int64))
    if kind == "host_c":
        seqs, offs, lens = s["pinned"]
        p = gs.Context.params(**params)
        gs.check(gs.lib().gs_seed(s["context"].h, ctypes.c_void_p(seqs.data_ptr()),
                                  ctypes.c_void_p(offs.data_ptr()),
                                  ctypes.c_void_p(lens.data_ptr()), lens.numel(), ctypes.byref(p)))
        return _host_result(s)
    if kind in ("device", "graph", "text"):
        seqs, offs, lens = s["on_device"]
        with torch.cuda.stream(s["stream"]):
            s["context"].seed_device(seqs.data_ptr(), offs.data_ptr(), lens.data_ptr(),
                                     lens.numel(), graph=kind == "graph", **params)
            if kind != "text":
                return _device_result(s)
            pointer, n = s["context"].text_device(1, params["smem"])
            v = _device_view(s["context"], pointer, (n,), "|u1", torch.uint8)
            return _kept(s["own"], "text", s["room"]["text"], v)
    if kind == "serve":
        server = s["server"]
        ids = [server.submit(*r) for r in s["requests"]]
        for i in ids:
            gs.check(server.wait(i))
        return [_of_result(server.result(i)[0], own, room)
                for i, own, room in zip(ids, s["own"], s["room"])]
    index = gs.build_index(s["codes"], sa_intv=7)
    ctx = gs.Context(index)
    r = ctx.seed(*s["reads"], **params)
    out = _of_result(r, s["own"], s["room"])
    info = index.info()
    out["header"] = np.array([info.seq_len, info.primary, info.n_sa, *info.L2], np.int64)
    ctx.close()
    index.close()
    return out


def work(c):
    """Bytes: the reads in, one 32-byte index sector per read position (both
    strands' matches that start there), and the results out, taken as four
    32-byte seeds with a position each and the two offsets a read."""
    reads = int(_sizes(c).sum()) if c["kind"] == "serve" else c["reads"]
    n = reads * (33 * _mean(c["lengths"]) + 12 + 4 * 36 + 16)
    if c["kind"] == "text":
        n += reads * 300                       # the records
    if c["kind"] == "build":
        # codes in, suffix array, occurrence blocks and samples out
        n += c["bases"] * (1 + 4 + 0.5 + 4 / 7)
    return {"bytes": float(n), "flops": 0.0}


def exact(c, seed):
    """Every output is whole numbers: nothing is rounded."""
    return None

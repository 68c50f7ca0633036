"""Workloads of the build path, called as a program calls the Python binding.

One case is one call (or one pair of calls) through the public entry points:

* ``build``   Engine.build: a collection resident in HBM, outputs left in HBM.
* ``host``    Engine.build: pinned host sequences in, host outputs out (what one
              serving request does).
* ``dropin``  Engine.phase1 + Engine.phase2: FASTA files in, bucket files
              between, frag_unitigs.bin and .color_sets out.
* ``files``   Engine.build_files: gzip FASTA files in, frag_unitigs.bin and
              .color_sets out, the buckets kept in HBM.
* ``seed``    Engine.stitch_seed: round 0 of the stitch from frag bytes in host
              memory to the round-0 files.
* ``server``  Server: a burst of build requests submitted together, all waited
              for.

The collections come from the package's own generator with the shapes of its
presets (``small``, ``pangenome``, ``largek``, ``skewed``, ``serving``); a
case's ``genomes`` and ``scale`` (genome length relative to the preset's) set
its size.  Files live in /dev/shm where there is one with room, as in
bench.py, so that no case waits for a disk.
"""
import ctypes
import math
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cdbg-builder_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from cdbg_gpu import native, synth  # noqa: E402

# ------------------------------------------------------------------- the cases


def listed():
    return [
        # a toy collection, as in a first run or a unit test: launches and
        # host waits are all there is
        _case("build_tiny", "build", "small", genomes=4, scale=0.004, k=31, buckets=64),
        # plasmid-sized sequences at large k, an odd length
        _case("build_tiny_k63", "build", "pangenome", genomes=7, scale=0.0277, k=63, buckets=256),
        # the plain small configuration: 10 genomes of 5 Mbp, -b 10
        _case("build_small", "build", "small", genomes=10, scale=1.0, k=31, buckets=1024),
        # a k outside the two usual ones, ragged genome lengths
        _case("build_k21", "build", "serving", genomes=33, scale=0.61, k=21, buckets=1024),
        # a fifth of the pangenome configuration, -b 12: the largest
        _case("build_pangenome", "build", "pangenome", genomes=200, scale=1.0, k=31, buckets=4096),
        # the large-k configuration: repeats, 128-bit k-mers
        _case("build_largek", "build", "largek", genomes=60, scale=1.0, k=63, buckets=4096),
        # the skewed configuration: heavy-tailed buckets, -b 14
        _case("build_skewed", "build", "skewed", genomes=90, scale=1.0, k=31, buckets=16384),
        # one serving request of middling size, host memory to host memory
        _case("host_request", "host", "serving", genomes=25, scale=0.5, k=63, buckets=1024),
        # the drop-in pair on the small configuration's FASTA files
        _case("dropin_small", "dropin", "small", genomes=10, scale=0.5, k=31, buckets=1024),
        # gzip files end to end, many of them, each of genome size
        _case("files_gz", "files", "pangenome", genomes=130, scale=0.5, k=31, buckets=4096),
        # round 0 of the stitch from a build's frag bytes
        _case("seed_small", "seed", "pangenome", genomes=24, scale=0.5, k=31, buckets=1024),
        # a burst of requests of both k-mer widths on a shared GPU
        _case("server_burst", "server", "serving", genomes=12, scale=0.3, k=31, buckets=1024),
    ]


def _case(name, kind, shape, genomes, scale, k, buckets):
    return {"name": name, "kind": kind, "shape": shape, "genomes": genomes, "scale": scale, "k": k,
            "buckets": buckets}


# megabases of input a drawn case of each kind may have: from a toy to (below)
# the largest listed case of its kind
_RANGE = {"build": (0.05, 900.0), "host": (1.0, 120.0), "dropin": (0.5, 50.0), "files": (4.0, 310.0),
          "seed": (2.0, 57.0), "server": (4.0, 60.0)}
_WEIGHT = ("build",) * 6 + ("host",) * 2 + ("files",) * 2 + ("dropin", "seed", "server")
# how a shape's cost per base compares with the pangenome's (k = 63 doubles the
# k-mers' bytes; large-k draws stay within the large-k case's size)
_MAX_LARGEK = 290.0


def draw(rng):
    kind = rng.choice(_WEIGHT)
    lo, hi = _RANGE[kind]
    shape = rng.choice({"build": ("small", "pangenome", "largek", "skewed", "serving"),
                        "host": ("serving", "small"), "dropin": ("small", "pangenome"),
                        "files": ("pangenome", "small"), "seed": ("pangenome", "small"),
                        "server": ("serving",)}[kind])
    k = 63 if shape == "largek" else rng.choice((31, 31, 31, 63, 21, 45)) if kind in ("build", "host") else 31
    if k > 31:
        hi = min(hi, _MAX_LARGEK)
    if kind == "build" and shape == "skewed":
        hi = min(hi, 290.0)
    if shape == "largek":
        lo = max(lo, 4.0)
    mb = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    # that many bases over a log-uniform number of genomes, each of at most the
    # preset's own length
    length = _mean_len(shape) / 1e6
    least = max(2, math.ceil(mb / length))
    most = max(least, min({"files": 160, "server": 24}.get(kind, 300), int(mb / 0.004)))
    genomes = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
    scale = min(1.0, max(0.0003, round(mb / genomes / length, 5)))
    top = 6 if mb < 1 else 10 if mb < 100 else 12
    buckets = 1 << rng.randint(max(5, top - 3), min(14, top + 2))
    if rng.random() < 0.25:
        buckets -= rng.randint(1, buckets // 3)
    return {"kind": kind, "shape": shape, "genomes": genomes, "scale": scale, "k": k, "buckets": buckets}


def _mean_len(shape):
    d = synth.PRESETS[shape][0]
    a, b = d["len_min"], d["len_max"]
    return a if a == b else (b - a) / math.log(b / a)


# -------------------------------------------------------------------- the work


def _bases(case):
    """(input bases, SNPs, bases of distinct sequence) of a case's collection,
    as expected."""
    d = synth.PRESETS[case["shape"]][0]
    n, length = case["genomes"], _mean_len(case["shape"]) * case["scale"]
    inserted = 3000 * d.get("repeats_per_genome", 0)  # shared repeats keep their length at every scale
    snps = n * length * 0.5 * (d["div_min"] + d["div_max"])
    return n * (length + inserted), snps, d["len_max"] * case["scale"] + 3000 * d.get("repeat_pool", 0)


def _frag_bytes(case):
    """Expected bytes of the fragments, ~61 each at k = 31: a SNP opens about
    six of them, fewer where SNPs of many genomes crowd, and the distinct
    sequence is cut into one per super-k-mer."""
    _, snps, distinct = _bases(case)
    wide = 1.0 if 25 <= case["k"] <= 31 else 1.3 if case["k"] < 25 else 1.6
    return wide * (snps * (150.0 + 230.0 / (1 + 4 * snps / distinct)) + 6.5 * distinct)


def work(case):
    """Input bytes read once and (expected) output bytes written once; the
    color sets add about an eighth to the fragments."""
    out = 1.125 * _frag_bytes(case)
    inp = {"files": 0.36}.get(case["kind"], 1.0) * _bases(case)[0]
    if case["kind"] == "seed":  # frag bytes in; tigs (2-bit bases) and closed unitigs out
        inp, out = _frag_bytes(case), 0.6 * _frag_bytes(case)
    if case["kind"] == "server":
        inp, out = 3.5 * inp, 4.0 * out
    return {"bytes": inp + out, "flops": 0}


# ------------------------------------------------------------ inputs and handles

_handles = {}


def _stream():
    """The stream the program and its engine work on."""
    if "stream" not in _handles:
        _handles["stream"] = torch.cuda.Stream()
    return _handles["stream"]


def _engine():
    """The process's engine: a program keeps one per device."""
    if "engine" not in _handles:
        _handles["engine"] = native.Engine(0)
        _handles["engine"].set_stream(_stream().cuda_stream)
    return _handles["engine"]


def _server():
    if "server" not in _handles:
        _handles["server"] = native.Server(device=0, slots=3, hbm_budget=100 << 30)
    return _handles["server"]


def _scratch():
    """A fresh folder, gone with the state that holds it."""
    base = "/dev/shm" if os.path.isdir("/dev/shm") and shutil.disk_usage("/dev/shm").free > (16 << 30) else None
    return tempfile.TemporaryDirectory(prefix="cdbg_cases_", dir=base)


def _collection(case, seed, genomes=None):
    p, _, _, _ = synth.preset(case["shape"], seed=seed, scale=case["scale"])
    n = genomes or case["genomes"]
    seq, lens, per = synth.collection(p, n)
    off = np.zeros(len(lens) + 1, dtype=np.uint64)
    off[1:] = np.cumsum(lens)
    return seq, off, np.repeat(np.arange(n, dtype=np.uint32), per)


def _batch(seq, off, col, device):
    """(SeqBatch, the tensors it points into): in HBM, or in pinned memory."""
    keep = [torch.from_numpy(seq), torch.from_numpy(off.view(np.int64)), torch.from_numpy(col.view(np.int32))]
    keep = [t.cuda() if device else t.pin_memory() for t in keep]
    if device:
        torch.cuda.synchronize()
    return native.SeqBatch(keep[0].data_ptr(), len(seq), keep[1].data_ptr(), keep[2].data_ptr(), len(col),
                           1 if device else 0), keep


def _files(case, seed, folder, gzip_level):
    p, _, _, _ = synth.preset(case["shape"], seed=seed, scale=case["scale"])
    lst = synth.write_fasta(p, case["genomes"], os.path.join(folder, "in"), gzip_level=gzip_level)
    with open(lst) as f:
        return [line.strip() for line in f if line.strip()]


def _room(case):
    """Bytes a program sets aside for the fragments: their expected size with
    a margin."""
    return (int(2.0 * _frag_bytes(case)) + (1 << 18)) & ~7


def _buffers(room, device):
    """The program's own buffers for a build's outputs, which the engine only
    lends until its next call."""
    make = lambda n, t: torch.zeros(n, dtype=t, device="cuda" if device else "cpu", pin_memory=not device)  # noqa: E731
    return {"frag": make(room, torch.uint8), "words": make(room // 32, torch.int64),
            "offsets": make(room // 32, torch.int64)}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "k": case["k"], "buckets": case["buckets"], "genomes": case["genomes"], "room": _room(case)}
    if kind in ("build", "host"):
        s["engine"] = _engine()
        s["batch"], s["keep"] = _batch(*_collection(case, seed), device=kind == "build")
        s["out"] = _buffers(s["room"], kind == "build")
    elif kind in ("dropin", "files"):
        s["engine"] = _engine()
        s["dir"] = _scratch()
        s["files"] = _files(case, seed, s["dir"].name, 1 if kind == "files" else 0)
        s["tmp"] = os.path.join(s["dir"].name, "buckets")
        os.makedirs(s["tmp"])
        s["frag"] = os.path.join(s["dir"].name, "frag_unitigs.bin")
        s["sets"] = os.path.join(s["dir"].name, "out.color_sets")
    elif kind == "seed":
        s["engine"] = _engine()
        s["dir"] = _scratch()
        batch, keep = _batch(*_collection(case, seed), device=False)
        r = s["engine"].build(batch, case["k"], case["buckets"], case["genomes"])
        s["frag"] = _host(r.frag_bytes, r.frag_nbytes, native.c_u8p).copy()
    elif kind == "server":
        # a burst of six requests, their sizes a part of the case's each, the
        # widths alternating
        s["server"] = _server()
        s["requests"], s["out"] = [], []
        for i in range(6):
            n = max(2, case["genomes"] * (6 - i) // 6)
            k = case["k"] if i % 2 == 0 else 63
            batch, keep = _batch(*_collection(case, 16 * seed + i, n), device=False)
            s["requests"].append((batch, keep, k, n))
            s["out"].append(_buffers(_room(dict(case, genomes=n, k=k)), False))
    return s


# ------------------------------------------------------------------- the calls


class _DeviceArray:
    """Device memory of a build's result, for torch.as_tensor (no copy)."""

    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": kind, "version": 3}


def _host(ptr, n, kind):
    return np.ctypeslib.as_array(ctypes.cast(ptr, kind), (n,)) if n else np.zeros(0, np.uint8)


def _take(out, r):
    """The build's outputs into the program's buffers."""
    words = (r.class_bits + 63) // 64
    for name, ptr, n in (("frag", r.frag_bytes, r.frag_nbytes), ("words", r.class_words, words),
                         ("offsets", r.class_offsets, r.n_color_sets)):
        if n == 0:
            continue
        if out[name].is_cuda:
            src = torch.as_tensor(_DeviceArray(ptr, n, "|u1" if name == "frag" else "<i8"), device="cuda")
        elif name == "frag":
            src = torch.from_numpy(_host(ptr, n, native.c_u8p))
        else:
            src = torch.from_numpy(_host(ptr, n, native.c_u64p).view(np.int64))
        out[name][:n].copy_(src)


def _counts(r):
    return [r.n_kmers, r.n_distinct, r.n_fragments, r.n_color_sets, r.class_bits, r.frag_nbytes]


def _mapped(path, room):
    """A file's bytes, with zeros up to `room`."""
    size = os.path.getsize(path) if os.path.exists(path) else 0
    if size > room:
        raise ValueError("%s has %d bytes, more than %d" % (path, size, room))
    with open(path, "ab") as f:
        f.truncate(room)
    return np.memmap(path, dtype=np.uint8, mode="r")


def run(state):
    kind, k, B, n, room = state["kind"], state["k"], state["buckets"], state["genomes"], state["room"]
    if kind == "build":
        with torch.cuda.stream(_stream()):
            r = state["engine"].build(state["batch"], k, B, n, outputs_to_host=False)
            _take(state["out"], r)
        return dict(state["out"], counts=_counts(r))
    if kind == "host":
        r = state["engine"].build(state["batch"], k, B, n)
        _take(state["out"], r)
        return dict(state["out"], counts=_counts(r))
    if kind == "dropin":
        s1, unc = state["engine"].phase1(state["files"], k, B, state["tmp"])
        s2 = state["engine"].phase2(state["tmp"], B, k, n, state["frag"], state["sets"])
        return {"frag": _mapped(state["frag"], room), "sets": _mapped(state["sets"], room // 2), "bucket_bytes": unc,
                "counts": [s1.n_kmers, s1.n_records, s2.n_distinct, s2.n_fragments, s2.n_color_sets]}
    if kind == "files":
        r = state["engine"].build_files(state["files"], k, B, state["frag"], state["sets"])
        return {"frag": _mapped(state["frag"], room), "sets": _mapped(state["sets"], room // 2), "counts": _counts(r)}
    if kind == "seed":
        out = os.path.join(state["dir"].name, "round0")
        closed = os.path.join(state["dir"].name, "closed.bin")
        st = state["engine"].stitch_seed((state["frag"].ctypes.data, state["frag"].nbytes), k, out, num_buckets=48,
                                         closed_path=closed)
        return {"round0": [_mapped(os.path.join(out, "stitch_r0_b%d.bin" % b), room // 16 + (1 << 16))
                           for b in range(48)],
                "closed": _mapped(closed, room),
                "counts": [st["fragments"], st["routed"], st["closed_unitigs"], st["round0_bytes"]]}
    srv = state["server"]
    ids = [srv.submit(batch, kk, B, c) for batch, _, kk, c in state["requests"]]
    got = []
    for i, out in zip(ids, state["out"]):
        d = srv.wait(i)
        if d["status"] != 0:
            raise RuntimeError(d["error"])
        for name in ("frag", "words", "offsets"):
            x = np.frombuffer(d[name], dtype=np.uint8) if name == "frag" else d[name].view(np.int64)
            out[name][:len(x)].copy_(torch.from_numpy(x))
        got.append(dict(out, counts=d["n_fragments"]))
    return got

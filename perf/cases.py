"""The calls this framework is used for, as measurable cases.

Every mapping case runs against a seeded synthetic reference of the presets in
shmap_b200/synth.py (uniform5m: 5 Mbp; human31: 3.1 Gbp with satellite arrays
and repeats) whose index stays resident, as a mapping program or a service
keeps it, in one device context per process. The reads are drawn anew for every
seed, with the read presets' lengths and errors (hifi, ont, dense, fixed10k).
Host inputs lie in pinned memory, as the integration notes ask for.

A case's "do":
  sketch       one sequence's k-mers (Context.sketch)
  map          records of host reads (SketchIndex.map_reads)
  map_device   records of reads in device memory, left there (map_reads_device)
  map_paf      records and PAF text of host reads (SketchIndex.map_paf)
  serve        requests of mixed sizes and read kinds through a Server
  index        an index built from bases in host memory, and what it holds
  whole_run    reference FASTA and reads FASTA in, records out: the command line's work
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "shmap-rs_b200"))

import shmap_b200 as sb  # noqa: E402
from shmap_b200 import synth  # noqa: E402

MEAN_LEN = {"hifi": 23_000, "ont": 24_000, "dense": 15_000, "fixed10k": 10_000}


def _map(name, do, reads, n, r=0.01, theta=0.4, metric="Containment", ref="human31"):
    return {"name": name, "do": do, "ref": ref, "reads": reads, "n": n, "k": 25, "r": r, "theta": theta,
            "metric": metric}


def listed():
    return [
        # one read's sketch: the latency of the smallest entry point
        {"name": "sketch_one_read", "do": "sketch", "bases": 23_001, "k": 25, "r": 0.01},
        # one read, as an interactive caller or an adaptive-sampling loop maps it
        _map("map_one_read", "map", "hifi", 1),
        # a request of the size a sequencer's basecaller emits at once
        _map("map_request", "map", "hifi", 257),
        # the small plain configuration: 5 Mbp reference, 2,000 reads of 10 kb
        _map("map_uniform10k", "map", "fixed10k", 2_000, ref="uniform5m"),
        # a service slot's batch, already on the device
        _map("hifi_batch_device", "map_device", "hifi", 2_049),
        # the headline workload: 150,000 HiFi-like reads resident in HBM
        _map("hifi_full_device", "map_device", "hifi", 150_000),
        # ONT-like reads under the symmetric metric
        _map("ont_jaccard_device", "map_device", "ont", 30_001, theta=0.1, metric="Jaccard"),
        # dense sampling: ten times the k-mers a read, a fifth of the reads in satellite arrays
        _map("dense_device", "map_device", "dense", 12_500, r=0.10),
        # chain-aware scoring of the same reads
        _map("hifi_lcs_device", "map_device", "hifi", 15_000, metric="bucket_LCS"),
        # file-to-file mapping: reads in pinned host memory in, records and PAF text out
        _map("hifi_paf_host", "map_paf", "hifi", 30_000),
        # a resident service: requests of HiFi-like and ONT-like reads submitted at once, then collected
        {"name": "serve_mixed", "do": "serve", "ref": "human31", "requests": 12, "most": 1_024, "k": 25, "r": 0.01,
         "theta": 0.1, "metric": "Containment"},
        # a whole run from FASTA bytes: parse both files, index the reference, map the reads
        {"name": "whole_run", "do": "whole_run", "ref": "human31", "scale": 0.05, "reads": "hifi", "n": 4_000,
         "k": 25, "r": 0.01, "theta": 0.4, "metric": "Containment"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    do = rng.choice(["sketch", "map", "map", "map_device", "map_device", "map_device", "map_paf", "serve", "index",
                     "whole_run"])
    if do == "sketch":
        return {"do": do, "bases": _log_int(rng, 200, 3_000_000), "k": rng.choice([15, 21, 25, 31]),
                "r": rng.choice([0.01, 0.05, 0.1])}
    if do == "index":
        return {"do": do, "ref": "human31", "scale": round(0.002 * 20 ** rng.random(), 6), "k": rng.choice([15, 21, 25]),
                "r": rng.choice([0.01, 0.02, 0.1])}
    if do == "whole_run":
        return {"do": do, "ref": "human31", "scale": round(0.002 * 25 ** rng.random(), 6), "reads": "hifi",
                "n": _log_int(rng, 20, 5_000), "k": rng.choice([15, 25]), "r": 0.01, "theta": 0.4,
                "metric": "Containment"}
    if do == "serve":
        return {"do": do, "ref": "human31", "requests": rng.randint(2, 16), "most": _log_int(rng, 8, 2_048), "k": 25,
                "r": 0.01, "theta": 0.1, "metric": rng.choice(["Containment", "Jaccard"])}
    reads = rng.choice(["hifi", "hifi", "ont", "dense", "fixed10k"])
    most = {"hifi": 40_000, "ont": 30_000, "dense": 8_000, "fixed10k": 20_000}[reads]
    metric = rng.choice({"hifi": ["Containment", "Containment", "Jaccard", "bucket_SH", "bucket_LCS"],
                         "ont": ["Containment", "Jaccard"], "dense": ["Containment", "bucket_SH"],
                         "fixed10k": ["Containment", "Jaccard"]}[reads])
    if do == "map_paf" or metric == "bucket_LCS":
        most //= 4
    c = _map("", do, reads, _log_int(rng, 1, most), r=0.10 if reads == "dense" else 0.01,
             theta=0.1 if reads == "ont" else rng.choice([0.4, 0.6]), metric=metric,
             ref="uniform5m" if reads == "fixed10k" else "human31")
    del c["name"]
    return c


# ------------------------------------------------------- what a program keeps
_kept = {}


def _keep(key, make):
    """Made once per process: the context, the references and their indexes."""
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _ctx():
    return _keep("ctx", lambda: sb.Context(0))


def _genome(ref):
    return _keep(("genome", ref), lambda: synth.Genome(synth.REFS[ref]))


def _index(ref, k, r):
    def make():
        g = _genome(ref)
        return sb.SketchIndex(_ctx(), g.names, g.seq, g.seg_off, k, r)
    return _keep(("index", ref, k, r), make)


def _server(c):
    idx = _index(c["ref"], c["k"], c["r"])
    return _keep(("server", c["ref"], c["k"], c["r"], c["theta"], c["metric"]),
                 lambda: sb.Server(_ctx(), idx, _params(c), slots=2, hbm_budget=16 << 30))


def _params(c):
    return sb.Params(k=c["k"], h_frac=c["r"], theta=c["theta"], metric=c["metric"])


# --------------------------------------------------------------------- inputs
def _read_spec(kind, n, seed):
    s = synth.READS[kind]
    return synth.replace(s, n_reads=n, seed=s.seed + 1_000_003 * (int(seed) + 1))


def _pinned(a):
    t = torch.empty(max(1, a.nbytes), dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    out = t.numpy()[: a.nbytes]
    out[:] = a.view(np.uint8).reshape(-1)
    return out


def _fasta(names, seq, offs, width=100):
    """FASTA bytes with lines of `width` bases."""
    out = []
    for i, name in enumerate(names):
        s = seq[offs[i]:offs[i + 1]]
        full = len(s) // width * width
        lines = np.empty((full // width, width + 1), np.uint8)
        lines[:, :width] = s[:full].reshape(-1, width)
        lines[:, width] = 10
        out += [b">" + name.encode() + b"\n", lines.tobytes()]
        if full < len(s):
            out += [s[full:].tobytes(), b"\n"]
    return b"".join(out)


def _room(bases, r):
    """K-mers that `bases` bases at hash ratio r never exceed (a sketch's size is random)."""
    return min(bases, int(1.5 * bases * r) + 256)


def prepare(case, seed):
    do = case["do"]
    ctx = _ctx()
    if do == "sketch":
        rng = np.random.default_rng(int(seed))
        return {"do": do, "ctx": ctx, "k": case["k"], "r": case["r"],
                "seq": np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, case["bases"])].tobytes(),
                "room": _room(case["bases"], case["r"])}
    if do in ("index", "whole_run"):
        spec = synth.scaled(synth.REFS[case["ref"]], case["scale"], seed=1_000 + int(seed))
        g = synth.Genome(spec)
        s = {"do": do, "ctx": ctx, "names": g.names, "k": case["k"], "r": case["r"]}
        if do == "index":
            s.update(seq=_pinned(g.seq), off=g.seg_off, room=_room(len(g.seq), case["r"]))
            return s
        names, seq, offs = g.reads(_read_spec(case["reads"], case["n"], seed))
        s.update(params=_params(case), ref_fa=_fasta(g.names, g.seq, g.seg_off), reads_fa=_fasta(names, seq, offs))
        return s
    idx = _index(case["ref"], case["k"], case["r"])
    g = _genome(case["ref"])
    if do == "serve":
        reqs = []
        for i in range(case["requests"]):
            n = 1 + int((case["most"] - 1) * (0.5 + 0.618034 * i) % case["most"])  # sizes spread over 1 .. most
            _, seq, offs = g.reads(_read_spec(("hifi", "ont")[i % 2], n, 131 * int(seed) + i))
            reqs.append((_pinned(seq), offs))
        return {"do": do, "server": _server(case), "reqs": reqs}
    names, seq, offs = g.reads(_read_spec(case["reads"], case["n"], seed))
    s = {"do": do, "index": idx, "params": _params(case), "names": names, "offs": offs}
    if do == "map_device":
        d = torch.zeros(len(seq) + 32, dtype=torch.uint8, device="cuda")
        d[: len(seq)] = torch.from_numpy(seq).cuda()
        s.update(seq=d, out=torch.zeros((len(offs) - 1, 15), dtype=torch.float64, device="cuda"))
    else:
        s["seq"] = _pinned(seq)
        if do == "map_paf":
            s["text"] = np.zeros(640 * case["n"] + 4096, np.uint8)
    return s


# ----------------------------------------------------------------------- runs
def _fields(rec):
    """A record array as its scores (f64) and its whole-number fields (int32)."""
    flat = rec.view(np.uint8).reshape(len(rec), sb.RECORD_DTYPE.itemsize)
    return {"scores": flat[:, :24].copy().view(np.float64), "fields": flat[:, 24:].copy().view(np.int32)}


def _kmers(room, r, h, strand, **more):
    """Arrays of one entry a k-mer at a length that does not depend on the inputs: -1 past the last."""
    out = {}
    for name, a in {"r": r, "h": h.view(np.int64), "strand": strand.view(np.int8), **more}.items():
        out[name] = np.full(room, -1, a.dtype)
        out[name][: len(a)] = a
    return out


def run(state):
    do = state["do"]
    if do == "sketch":
        return _kmers(state["room"], *state["ctx"].sketch(state["seq"], state["k"], state["r"]))
    if do == "map":
        return _fields(state["index"].map_reads(state["params"], state["seq"], state["offs"]))
    if do == "map_device":
        out = state["out"]
        state["index"].map_reads_device(state["params"], state["seq"].data_ptr(), state["offs"], out.data_ptr())
        return {"scores": out[:, :3], "fields": out.view(torch.int32)[:, 6:]}
    if do == "map_paf":
        text, rec = state["index"].map_paf(state["params"], state["seq"], state["offs"], state["names"])
        text = np.frombuffer(text.encode(), np.uint8)
        state["text"][: len(text)] = text
        return {"text": state["text"], **_fields(rec)}
    if do == "serve":
        tickets = [state["server"].submit(seq, offs) for seq, offs in state["reqs"]]
        return [_fields(state["server"].poll(t)[0]) for t in tickets]
    if do == "index":
        idx = sb.SketchIndex(state["ctx"], state["names"], state["seq"], state["off"], state["k"], state["r"])
        r, h, strand = (np.concatenate(a) for a in zip(*(idx.segment(i)[:3] for i in range(len(state["names"])))))
        return {"stats": list(idx.stats().values()), **_kmers(state["room"], r, h, strand, count=idx.count(h))}
    ref = sb.DeviceFasta(state["ctx"], state["ref_fa"])
    idx = sb.SketchIndex.from_device_fasta(state["ctx"], ref, state["k"], state["r"])
    reads = sb.DeviceFasta(state["ctx"], state["reads_fa"])
    rec = idx.map_device_fasta(state["params"], reads)
    return {"stats": list(idx.stats().values()), "offs": reads.offs, **_fields(rec)}


def work(case):
    """Every base read once, every k-mer's index entry read once (a 32-byte sector) and every result written once."""
    do = case["do"]
    if do == "sketch":
        return {"bytes": case["bases"] + 13 * case["bases"] * case["r"], "flops": 0}
    if do in ("index", "whole_run"):
        ref = synth.REFS[case["ref"]].total_bases * case["scale"]
        n = ref + 40 * ref * case["r"]
        if do == "whole_run":
            bases = case["n"] * MEAN_LEN[case["reads"]]
            n += bases * (1 + 32 * case["r"]) + 120 * case["n"]
        return {"bytes": n, "flops": 0}
    n = case["requests"] * (case["most"] + 1) / 2 if do == "serve" else case["n"]
    bases = n * (MEAN_LEN["hifi"] if do == "serve" else MEAN_LEN[case["reads"]])
    return {"bytes": bases * (1 + 32 * case["r"]) + (600 if do == "map_paf" else 120) * n, "flops": 0}


# --------------------------------------------------------------------- checks
def exact(case, seed):
    """The sketch, from ntHash's definition. The other outputs are whole numbers and quotients of whole numbers that
    only the complete mapping path gives; plain numpy would take minutes for the smallest of those cases."""
    if case["do"] != "sketch":
        return None
    k = case["k"]
    word = {65: 0x3C8BFBB395C60474, 67: 0x3193C18562A02B4C, 71: 0x20323ED082572324, 84: 0x295549F54BE24456}
    rng = np.random.default_rng(int(seed))
    seq = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, case["bases"])]
    fw, rc = np.zeros(256, np.uint64), np.zeros(256, np.uint64)
    for b, comp in ((65, 84), (67, 71), (71, 67), (84, 65)):
        fw[b], rc[b] = word[b], word[comp]
    n = len(seq) - k + 1

    def rol(x, s):
        s %= 64
        return x if s == 0 else (x << np.uint64(s)) | (x >> np.uint64(64 - s))

    f, c = np.zeros(n, np.uint64), np.zeros(n, np.uint64)
    for i in range(k):
        f ^= rol(fw[seq[i:i + n]], k - 1 - i)
        c ^= rol(rc[seq[i:i + n]], i)
    h = f ^ c
    at = np.flatnonzero(h <= np.uint64(int(case["r"] * float(2 ** 64 - 1))))
    return _kmers(_room(case["bases"], case["r"]), (at + k - 1).astype(np.int32), h[at],
                  (f[at] > c[at]).astype(np.uint8))

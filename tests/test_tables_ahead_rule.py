"""Which reads are put down for a second bucket table before their
contributions: array reads with a processed seed and 16 hits for each of 512
slots, no plain ones, no array reads of few seeds or few hits, and no more
than three quarters of the spare tables."""
import ctypes

import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


def _ahead(ctx):
    f = sb.lib().shm_internal_ctx_state
    f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_void_p, ctypes.c_int32]
    return f(ctx.h, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("reads, copies, spare, ahead", [
    ("array", 234, None, 5),     # all five
    ("plain", 234, None, 0),     # a hit a seed
    ("short", 234, None, 0),     # 186 seeds
    ("array", 6, None, 0),       # six hits a seed
    ("array", 234, 8192, 1),     # two spare tables, one of them at most ahead
    ("array", 234, 4096, 0),     # one spare table
    ("array", 234, 0, 0)])       # none
def test_reads_put_down(gpu_ctx, monkeypatch, reads, copies, spare, ahead):
    k, rng = 15, np.random.default_rng(copies)
    dna = lambda n: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)]  # noqa: E731
    array = np.tile(dna(1711), copies)
    hit = rng.random(len(array)) < 0.01
    array[hit] = dna(int(hit.sum()))
    plain = dna(500_000)
    ref = [("a", array.tobytes()), ("p", plain.tobytes())]
    n = 600 if reads == "short" else 2_500
    src = plain if reads == "plain" else array
    seq, offs = pack([src[s:s + n].tobytes() for s in range(0, 7_500, 1_500)])
    if spare is not None:
        monkeypatch.setenv("SHMAP_BT_SPARE_SLOTS", str(spare))
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 0.5), O.Index.from_records(ref, k, 0.5)
    kw = dict(k=k, h_frac=0.5, theta=0.4)
    before = _ahead(gpu_ctx)
    rec = g.map_reads(sb.Params(**kw), seq, offs)
    assert _ahead(gpu_ctx) - before == ahead
    mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
    assert not mm, mm
    g.close()

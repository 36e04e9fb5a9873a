"""What a context keeps between calls: sketch tables, which sketching at another
k than the mapping's must not make anew at every change."""
import ctypes

import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches, xorshift_dna

pytestmark = pytest.mark.gpu


def _state(ctx, what):
    f = sb.lib().shm_internal_ctx_state
    f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_void_p, ctypes.c_int32]
    return f(ctx.h, what)


def test_tables_of_two_k():
    ctx, ref = sb.Context(0), xorshift_dna(11, 60_000)
    idx = sb.SketchIndex.from_records(ctx, [("r", ref)], 25, 0.05)
    seq, offs = pack([ref[s:s + 2_000] for s in range(0, 50_000, 1_000)])
    p = sb.Params(k=25, h_frac=0.05, theta=0.4)
    want = idx.map_reads(p, seq, offs)
    assert _state(ctx, 0) == 1  # the index's, which the mapping uses too
    for _ in range(4):
        for k in (15, 17):
            got, sk = ctx.sketch(ref, k, 0.05), O.sketch(ref, k, 0.05)
            assert all(np.array_equal(a, b) for a, b in zip(got, sk))
        assert not record_mismatches(idx.map_reads(p, seq, offs), want)
    # the mapping's once more (the index's made way for the sketches'), then only those of 15 and 17
    assert _state(ctx, 0) == 1 + 8 + 1
    for _ in range(4):
        ctx.sketch(ref, 17, 0.05)
        assert not record_mismatches(idx.map_reads(p, seq, offs), want)
    assert _state(ctx, 0) == 1 + 8 + 1
    idx.close()
    ctx.close()

"""Sketches larger than the context's pinned staging come back in pieces of 2^19
windows (csrc/shm_capi.cu): every window, at each side of the pieces' ends, and
the block stays small."""
import ctypes

import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import lcg_dna

pytestmark = pytest.mark.gpu

PIECE, K = 1 << 19, 25


@pytest.mark.parametrize("windows", [2 * PIECE - 1, 2 * PIECE, 2 * PIECE + 1, 3 * PIECE, 3 * PIECE + 1, 4 * PIECE + 7,
                                     8 * PIECE, 8 * PIECE + 1, 10 * PIECE + 13])
def test_sketches_in_pieces(windows):
    ctx = sb.Context(0)
    seq = lcg_dna(windows, windows + K - 1)
    for ratio in (1.0, 0.3):
        got, want = ctx.sketch(seq, K, ratio), O.sketch(seq, K, ratio)
        assert all(len(a) == len(b) and np.array_equal(a, b) for a, b in zip(got, want))
        assert ratio < 1.0 or len(got[0]) == windows
    f = sb.lib().shm_internal_ctx_state
    f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_void_p, ctypes.c_int32]
    assert f(ctx.h, 1) <= 16 << 20
    ctx.close()


def test_more_windows_than_expected():
    """A repeat that is selected whole: the count passes what came back first."""
    ctx = sb.Context(0)
    unit = lcg_dna(5, 400)
    r, h, s = O.sketch(unit + unit, 15, 0.01)
    at = int(r[0]) - 15 + 1
    seq = lcg_dna(6, 50) + (unit + unit)[at:at + 15] * 300_000
    got, want = ctx.sketch(seq, 15, 0.01), O.sketch(seq, 15, 0.01)
    assert len(want[0]) > 0.04 * len(seq)
    assert all(len(a) == len(b) and np.array_equal(a, b) for a, b in zip(got, want))
    ctx.close()

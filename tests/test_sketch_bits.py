"""The bit-plane read sketch against the oracle, at the edges of its tiles
(32 sub-runs of 120 windows), of its k range and of its threshold range."""
import ctypes

import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from test_gpu_parity import _read_sketches

TILE = 32 * 120


def _at_offset(reads, lead, k, r, packed):
    """_read_sketches with the first read `lead` bases into the device copy."""
    f = sb.lib().shm_internal_sketch_reads
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32, ctypes.c_double,
                  ctypes.c_int] + [ctypes.c_void_p] * 4
    seq = np.frombuffer(b"G" * lead + b"".join(reads), np.uint8)
    offs = lead + np.concatenate([[0], np.cumsum([len(x) for x in reads])]).astype(np.int64)
    caps = np.array([max(0, len(x) - k + 1) for x in reads], np.uint64)
    cap_off = np.concatenate([[0], np.cumsum(caps)]).astype(np.uint64)
    h, rs = np.zeros(int(cap_off[-1]) + 1, np.uint64), np.zeros(int(cap_off[-1]) + 1, np.uint32)
    cnt = np.zeros(len(reads), np.uint32)
    assert f(0, seq.ctypes.data, offs.ctypes.data, len(reads), k, r, packed, cap_off.ctypes.data, h.ctypes.data,
             rs.ctypes.data, cnt.ctypes.data) == 0
    out = []
    for i in range(len(reads)):
        a, m = int(cap_off[i]), int(cnt[i])
        o = np.argsort(rs[a:a + m] >> 1)
        out.append(((rs[a:a + m][o] >> 1).astype(np.int32), h[a:a + m][o], (rs[a:a + m][o] & 1).astype(np.uint8)))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("k", [14, 15, 16, 24, 25, 28, 29, 32, 33])
@pytest.mark.parametrize("r", [0.26, 0.25, 0.1, 0.01, 1e-4])
def test_tile_edges(gpu_ctx, k, r):
    rng = np.random.default_rng(k)

    def dna(n):
        return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()

    sets = [[dna(L)] for L in (k, 119, 120, 121, TILE - 1, TILE, TILE + 1, TILE + k - 2, TILE + k - 1, TILE + k,
                               2 * TILE + 7)]
    sets.append([dna(int(n)) for n in rng.integers(0, 3 * k, 400)])  # many reads a tile
    sets.append([dna(5 * TILE + 1), b"", dna(k - 1), dna(TILE)])
    sets.append([b"A" * TILE + dna(300), b"ACGT" * 1500, (b"CG" * 3000).lower()])  # every window alike
    s = bytearray(dna(6 * TILE))
    s[TILE + 119] = ord("N")                      # one masked base at a sub-run's end
    s[3 * TILE - 1:3 * TILE + 1] = b"nR"          # on a tile's edge
    s[4 * TILE:5 * TILE + 50] = b"N" * (TILE + 50)  # a whole tile
    sets.append([bytes(s), dna(700)])
    for n, reads in enumerate(sets):
        for packed in (0, 1):
            got = _read_sketches(reads, k, r, packed)
            for i, x in enumerate(reads):
                assert all(np.array_equal(a, b) for a, b in zip(got[i], O.sketch(x, k, r))), (n, packed, i, len(x))


@pytest.mark.gpu
@pytest.mark.parametrize("lead", [1, 2, 3, 5, 15, 17, 30, 31])
def test_any_first_base(gpu_ctx, lead):
    rng = np.random.default_rng(lead)
    reads = [np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes() for n in (2 * TILE + 3, 50, 3811)]
    for packed in (0, 1):
        got = _at_offset(reads, lead, 25, 0.05, packed)
        for i, x in enumerate(reads):
            assert all(np.array_equal(a, b) for a, b in zip(got[i], O.sketch(x, 25, 0.05))), (packed, i)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [14, 15, 25, 28, 32, 33])
@pytest.mark.parametrize("r", [1.0, 0.1, 0.01])
def test_ordered_edges(gpu_ctx, k, r):
    """One sequence's sketch and an index's segments, in order: at tile edges,
    with masked bases, with segments shorter than k, and with far more k-mers
    than a random sequence of the length would have."""
    rng = np.random.default_rng(k)

    def dna(n):
        return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()

    masked = bytearray(dna(4 * TILE))
    masked[TILE + 119] = ord("N")
    masked[2 * TILE - 1:2 * TILE + 1] = b"nR"
    masked[3 * TILE:] = b"N" * TILE
    rich = next(u for u in (dna(40) for _ in range(400)) if len(O.sketch(u * 3, k, 0.01)[0]) > 3)  # selected once a copy
    seqs = [dna(n) for n in (k, 120 + k - 1, TILE, TILE + k, 7 * TILE + 5)] + [bytes(masked), (rich * 2000)[:70001]]
    for x in seqs:
        got, want = gpu_ctx.sketch(x, k, r, 7), O.sketch(x, k, r, 7)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), len(x)
    recs = [(f"s{i}", x) for i, x in enumerate([dna(3), *seqs, b"", dna(k - 1), dna(2 * TILE + 1)])]
    idx = sb.SketchIndex.from_records(gpu_ctx, recs, k, r)
    for i, (_, x) in enumerate(recs):
        assert all(np.array_equal(a, b) for a, b in zip(idx.segment(i)[:3], O.sketch(x, k, r))), i
    idx.close()

"""bucket_LCS by bit vectors against the oracle: reads whose k-mer counts lie
at the edges of the vector widths, from unique and from tandem sequence, both
strands, and the two-pass refinement with all bucket variants."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


def _revcomp(s):
    return s[::-1].translate(bytes.maketrans(b"ACGT", b"TGCA"))


def _mutate(s, rng, rate):
    b = bytearray(s)
    for i in np.flatnonzero(rng.random(len(b)) < rate):
        b[i] = b"ACGT"[rng.integers(0, 4)]
    return bytes(b)


@pytest.mark.gpu
@pytest.mark.parametrize("opts", [{}, {"no_bucket_pruning": True}, {"one_sweep": True}, {"abs_pos": True}])
@pytest.mark.parametrize("m", [6, 511, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097])
def test_vector_widths(gpu_ctx, m, opts):
    k, rng = 15, np.random.default_rng(m)
    dna = lambda n: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()  # noqa: E731
    unit, long_unit = dna(37), dna(700)
    tandem = _mutate(unit * 300, rng, 0.01) + _mutate(long_unit * 12, rng, 0.02)
    ref = [("a", dna(9000) + tandem + dna(6000)), ("b", _revcomp(tandem) + dna(9000))]
    n = m + k - 1
    reads = [ref[0][1][2000:2000 + n], _revcomp(ref[0][1][2500:2500 + n])]
    for at in (8990, 11000, 9000 + 37 * 300 - n // 2):
        reads += [_mutate(ref[0][1][at:at + n], rng, 0.01), _revcomp(ref[0][1][at:at + n])]
    reads += [(unit * (n // 37 + 1))[:n], (b"AC" * n)[:n], dna(n)]
    seq, offs = pack(reads)
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 1.0), O.Index.from_records(ref, k, 1.0)
    for theta in (0.0, 0.4):
        kw = dict(k=k, h_frac=1.0, theta=theta, metric="bucket_LCS", **opts)
        rec = g.map_reads(sb.Params(**kw), seq, offs)
        mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
        assert not mm, (theta, mm)
    assert set(rec["sketch_size"]) == {m}
    g.close()

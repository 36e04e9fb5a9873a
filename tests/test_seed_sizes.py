"""Seed preparation at the edges of its size classes (a warp, then a CTA of
growing size, then global scratch), from unique and repeated sequence, against
the oracle's records."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["Containment", "bucket_SH"])
@pytest.mark.parametrize("m", [256, 257, 512, 513, 1024, 1025, 1100, 2048, 2049, 4096, 4097, 8192, 8193])
def test_size_class_edges(gpu_ctx, m, metric):
    k, rng = 17, np.random.default_rng(m)
    dna = lambda n: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()  # noqa: E731
    n = m + k - 1
    unique, unit = dna(3 * n + 500), dna(211)
    ref = [("u", unique), ("t", unit * (n // 211 + 60)), ("v", unique[n // 2:n // 2 + n] + dna(400))]
    half = unique[100:100 + n // 2]
    reads = [unique[50:50 + n],                                     # every k-mer once
             (unit * (n // 211 + 1))[:n],                           # few hashes, many occurrences each
             half + (unit * (n // 211 + 1))[:n - len(half)],        # both
             b"A" * n,                                              # one hash
             dna(n)]                                                # no hits
    seq, offs = pack(reads)
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 1.0), O.Index.from_records(ref, k, 1.0)
    for theta in (0.0, 0.5):
        kw = dict(k=k, h_frac=1.0, theta=theta, metric=metric)
        rec = g.map_reads(sb.Params(**kw), seq, offs)
        mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
        assert not mm, (theta, mm)
    assert set(rec["sketch_size"]) == {m}
    g.close()

"""Reads of tandem arrays in the seed preparation of 1,025 to 8,192 k-mers: a few
hashes hundreds of times each, two of them in one bucket of the hash order, which
must give the oracle's records and cost about what other reads cost."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches, xorshift_dna

pytestmark = pytest.mark.gpu

K = 17
UNIT = b"TGTGTTGGAC"  # two of the ten k-mers of its array share a bucket of 8,192 or fewer


@pytest.mark.parametrize("m, buckets", [(1_025, 2_048), (2_000, 2_048), (4_000, 4_096), (8_000, 8_192)])
def test_two_hashes_in_one_bucket(gpu_ctx, m, buckets):
    n = m + K - 1
    shared = {int(h) * buckets >> 64 for h in O.sketch(UNIT * 3, K, 1.0)[1]}
    assert len(shared) == 9
    array, other = (UNIT * (n // 10 + 1))[:n], xorshift_dna(m, n)
    ref = [("a", xorshift_dna(1, 3_000) + UNIT * 900 + xorshift_dna(2, 3_000)), ("b", xorshift_dna(m, n + 500))]
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, K, 1.0), O.Index.from_records(ref, K, 1.0)
    seq, offs = pack([array, other, array[:n // 2] + other[:n - n // 2]])
    for metric in ("Containment", "bucket_SH"):
        kw = dict(k=K, h_frac=1.0, theta=0.3, metric=metric)
        mm = record_mismatches(g.map_reads(sb.Params(**kw), seq, offs), o.map_reads(O.params(**kw), seq, offs))
        assert not mm, mm
    ms = []
    for read in (array, other):
        seq, offs = pack([read])
        for rep in range(15):
            if rep == 5:
                gpu_ctx.set_timing(True)
            g.map_reads(sb.Params(k=K, h_frac=1.0, theta=0.9, metric="bucket_SH"), seq, offs)
        ms.append(gpu_ctx.stage_times()["seedprep"][0])
        gpu_ctx.set_timing(False)
    assert ms[0] < 3 * ms[1], ms
    g.close()

"""The sweep's second threshold, best * (1 - min_diff), where it is not above
theta * (1 - min_diff): min_diff above 1, with candidates that score zero or
whose window is empty (absolute positions). Records equal the oracle's."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches, xorshift_dna


@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["Containment", "Jaccard", "bucket_SH", "bucket_LCS"])
@pytest.mark.parametrize("abs_pos", [False, True])
@pytest.mark.parametrize("min_diff", [1.0, 1.5, 3.0])
def test_low_second_threshold(gpu_ctx, metric, abs_pos, min_diff):
    k, r = 15, 0.05
    dna = xorshift_dna(5, 60_000)
    # copies of one stretch in both segments, so that reads have several candidates
    ref = [("a", dna[:30_000] + dna[4_000:9_000] + dna[30_000:40_000]), ("b", dna[40_000:60_000] + dna[2_000:12_000])]
    reads = [dna[s:s + n] for s in range(3_000, 10_000, 500) for n in (600, 1_500, 2_900)] + [dna[45_000:47_000]]
    seq, offs = pack(reads)
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, r), O.Index.from_records(ref, k, r)
    for theta in (0.0, 0.3):
        for nbp in (False, True):
            kw = dict(k=k, h_frac=r, theta=theta, metric=metric, min_diff=min_diff, abs_pos=abs_pos,
                      no_bucket_pruning=nbp)
            rec = g.map_reads(sb.Params(**kw), seq, offs)
            mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
            assert not mm, (theta, nbp, mm)
    g.close()

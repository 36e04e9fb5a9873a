"""Extension on both sides of its rule (the warps of a block in step from 8
bucket jobs a read on): reads of repeat arrays whose buckets all extend, alone
and diluted with reads that have none, against the oracle's records."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["Containment", "Jaccard", "bucket_SH"])
@pytest.mark.parametrize("plain,in_step", [(0, True), (3, True), (400, False)])
def test_jobs_a_read(gpu_ctx, plain, in_step, metric):
    k, rng = 15, np.random.default_rng(plain + 7)
    dna = lambda n: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)]  # noqa: E731
    unit = dna(171)
    array = np.tile(unit, 240)
    hit = rng.random(len(array)) < 0.01
    array[hit] = dna(int(hit.sum()))
    flank = dna(9000)
    ref = [("a", (flank.tobytes() + array.tobytes())), ("b", array[5000:25000].tobytes() + dna(700).tobytes())]
    reads = [array[s:s + n].tobytes() for s, n in ((0, 1500), (3001, 1731), (9000, 2333), (20000, 900), (30011, 1200))]
    reads += [dna(700 + i).tobytes() for i in range(plain)]
    seq, offs = pack(reads)
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 0.5), O.Index.from_records(ref, k, 0.5)
    kw = dict(k=k, h_frac=0.5, theta=0.4, metric=metric)
    gpu_ctx.set_timing(False)
    before = gpu_ctx.work_stats()["bucket_jobs"]
    rec = g.map_reads(sb.Params(**kw), seq, offs)
    jobs = gpu_ctx.work_stats()["bucket_jobs"] - before
    assert (jobs >= 8 * len(reads)) == in_step, jobs
    mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
    assert not mm, mm
    g.close()

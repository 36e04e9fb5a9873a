"""Reads put down for a second bucket table before their contributions (a
capped first table, a processed seed and 16 hits or more for each of its
slots), with many and with few distinct buckets, among reads on the other side of the rule, against
the oracle's records."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["Containment", "bucket_SH"])
@pytest.mark.parametrize("array_len", [400_000, 60_000])
def test_reads_of_repeat_arrays(gpu_ctx, array_len, metric):
    k, rng = 15, np.random.default_rng(array_len)
    dna = lambda n: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)]  # noqa: E731
    array = np.tile(dna(1711), array_len // 1711 + 1)[:array_len]
    hit = rng.random(len(array)) < 0.01
    array[hit] = dna(int(hit.sum()))
    plain = dna(900_000 - array_len)
    ref = [("a", array.tobytes()), ("p", plain.tobytes())]
    reads = [array[s:s + n].tobytes() for s, n in ((0, 2400), (5000, 2731), (9000, 2433), (12000, 600), (3011, 5200))]
    reads += [plain[s:s + 700].tobytes() for s in range(0, 30_000, 3_000)]
    seq, offs = pack(reads)
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 0.5), O.Index.from_records(ref, k, 0.5)
    kw = dict(k=k, h_frac=0.5, theta=0.4, metric=metric)
    before = gpu_ctx.work_stats()["second_tables"]
    rec = g.map_reads(sb.Params(**kw), seq, offs)
    assert gpu_ctx.work_stats()["second_tables"] > before
    mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
    assert not mm, mm
    g.close()

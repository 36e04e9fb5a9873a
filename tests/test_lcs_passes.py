"""bucket_LCS refines in two passes, the reads' leads first, only where that
leaves candidates out: not under absolute positions, and not the reads of more
than 4,096 k-mers, whose windows are too long to wait for one another."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import pack, record_mismatches


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2_000, 4_110, 4_111])
@pytest.mark.parametrize("opts, all_refined", [({}, False), ({"abs_pos": True}, True)])
def test_candidates_refined(gpu_ctx, n, opts, all_refined):
    k, rng = 15, np.random.default_rng(n)
    dna = lambda m: np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, m)]  # noqa: E731
    stretch = dna(9_000)
    copies = []
    for rate in (0.0, 0.03, 0.05, 0.06, 0.07, 0.08):  # ever worse copies of it
        c = stretch.copy()
        hit = rng.random(len(c)) < rate
        c[hit] = dna(int(hit.sum()))
        copies += [dna(3_000), c]
    ref = [("a", np.concatenate(copies).tobytes())]
    seq, offs = pack([stretch[s:s + n].tobytes() for s in range(0, 4_800, 400)])
    g, o = sb.SketchIndex.from_records(gpu_ctx, ref, k, 1.0), O.Index.from_records(ref, k, 1.0)
    kw = dict(k=k, h_frac=1.0, theta=0.2, min_diff=0.02, metric="bucket_LCS", **opts)
    before = gpu_ctx.work_stats()
    rec = g.map_reads(sb.Params(**kw), seq, offs)
    after = gpu_ctx.work_stats()
    mm = record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs))
    assert not mm, mm
    cands, refined = (after[f] - before[f] for f in ("candidates", "refined_candidates"))
    assert cands > len(rec)
    all_refined = all_refined or n - k + 1 > 4_096
    assert refined == cands if all_refined else refined < cands, (refined, cands)
    g.close()

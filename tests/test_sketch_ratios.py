"""The sketch at high hash ratios, where the rolling kernels take what the bit
planes take below: on both sides of every line of that rule the oracle's
k-mers, and for a short read no cost out of proportion."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from test_gpu_parity import _read_sketches

RATIOS = [0.25, 0.2501, 1 / 3, 0.334, 0.5, 0.501, 1.0]


def _dna(rng, n):
    return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("r", RATIOS)
def test_reads_on_both_sides(gpu_ctx, r):
    k, rng = 25, np.random.default_rng(7)
    # (reads, their length): a tile, 500 and 2,000 bases a read, 100,000 and 300,000 in all, and one more
    for n, length in ((1, 3840), (1, 3841), (9, 500), (9, 501), (1, 100_000), (1, 100_001), (151, 2000), (150, 2000),
                      (151, 2001), (1, 300_000), (1, 300_001)):
        reads = [_dna(rng, length) for _ in range(n)]
        reads[0] = reads[0][:700] + b"N" + reads[0][701:]
        for packed in (0, 1):
            got = _read_sketches(reads, k, r, packed)
            for i in {0, n // 2, n - 1}:
                assert all(np.array_equal(a, b) for a, b in zip(got[i], O.sketch(reads[i], k, r))), (n, length, packed)


@pytest.mark.gpu
@pytest.mark.parametrize("r", RATIOS)
def test_in_order_on_both_sides(gpu_ctx, r):
    k, rng = 25, np.random.default_rng(8)
    for n in (k, 150, 3841, 30_011):
        x = _dna(rng, n)
        assert all(np.array_equal(a, b) for a, b in zip(gpu_ctx.sketch(x, k, r), O.sketch(x, k, r))), n
    recs = [(f"s{i}", _dna(rng, n)) for i, n in enumerate((9_001, 3, 4_000))]
    idx = sb.SketchIndex.from_records(gpu_ctx, recs, k, r)
    for i, (_, x) in enumerate(recs):
        assert all(np.array_equal(a, b) for a, b in zip(idx.segment(i)[:3], O.sketch(x, k, r))), i
    idx.close()


@pytest.mark.gpu
def test_cost_of_a_short_read(gpu_ctx):
    """One read of 150 bases: its sketch stage at ratio 1 no more than eight
    times that at 0.2 (126 k-mers and 25; the planes took 17 times as long)."""
    import torch

    dna = np.frombuffer(_dna(np.random.default_rng(9), 20_000), np.uint8)
    d = torch.zeros(182, dtype=torch.uint8, device="cuda")
    d[:150] = torch.from_numpy(dna[5_000:5_150].copy()).cuda()
    out, offs, ms = torch.zeros(120, dtype=torch.uint8, device="cuda"), np.array([0, 150], np.int64), {}
    for r in (0.2, 1.0):
        idx = sb.SketchIndex(gpu_ctx, ["a"], dna, np.array([0, len(dna)], np.int64), 25, r)
        for rep in range(30):
            if rep == 10:
                gpu_ctx.set_timing(True)
            idx.map_reads_device(sb.Params(k=25, h_frac=r, theta=0.4), d.data_ptr(), offs, out.data_ptr())
        torch.cuda.synchronize()
        ms[r] = gpu_ctx.stage_times()["sketch"][0]
        gpu_ctx.set_timing(False)
        idx.close()
    assert ms[1.0] < 8 * ms[0.2], ms

"""The read sketch where every tile holds a base that is no letter: the same
k-mers (tests/test_sketch_bits.py), and no more than seven times the clean
reads' sketch stage (it rolls every window, about four times the
instructions)."""
import numpy as np
import pytest

import shmap_b200 as sb


@pytest.mark.gpu
def test_cost_of_marked_reads(gpu_ctx):
    import torch

    rng = np.random.default_rng(3)
    bases, n = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 60_000_000)], 3_000
    idx = sb.SketchIndex(gpu_ctx, ["a"], bases[:200_000], np.array([0, 200_000], np.int64), 25, 0.01)
    offs = np.arange(n + 1, dtype=np.int64) * (len(bases) // n)
    marked = bases.copy()
    marked[::500] = ord("N")
    out = torch.zeros(n * 120, dtype=torch.uint8, device="cuda")
    ms = {}
    for name, seq in (("clean", bases), ("marked", marked)):
        d = torch.zeros(len(seq) + 32, dtype=torch.uint8, device="cuda")
        d[: len(seq)] = torch.from_numpy(seq).cuda()
        for rep in range(13):
            if rep == 3:
                gpu_ctx.set_timing(True)
            idx.map_reads_device(sb.Params(k=25, h_frac=0.01, theta=0.4), d.data_ptr(), offs, out.data_ptr())
        torch.cuda.synchronize()
        ms[name] = gpu_ctx.stage_times()["sketch"][0] / 10
        gpu_ctx.set_timing(False)
    idx.close()
    assert ms["marked"] < 7 * ms["clean"], ms

"""Seed preparation of reads beyond the shared-memory classes (more than 8,192
k-mers), many at once: no more than ten times that of reads just below them,
which a CTA prepares on chip."""
import numpy as np
import pytest

import shmap_b200 as sb


@pytest.mark.gpu
def test_cost_beyond_the_classes(gpu_ctx):
    import torch

    rng, n, ms = np.random.default_rng(3), 300, {}
    dna = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 4_000_000)]
    idx = sb.SketchIndex(gpu_ctx, ["a"], dna[:200_000], np.array([0, 200_000], np.int64), 25, 0.1)
    out = torch.zeros(n * 120, dtype=torch.uint8, device="cuda")
    for length in (76_000, 95_000):  # about 7,600 and 9,500 k-mers
        at = rng.integers(0, len(dna) - length, n)
        d = torch.zeros(n * length + 32, dtype=torch.uint8, device="cuda")
        d[: n * length] = torch.from_numpy(np.concatenate([dna[a:a + length] for a in at])).cuda()
        offs = np.arange(n + 1, dtype=np.int64) * length
        for rep in range(8):
            if rep == 3:
                gpu_ctx.set_timing(True)
            idx.map_reads_device(sb.Params(k=25, h_frac=0.1, theta=0.9), d.data_ptr(), offs, out.data_ptr())
        torch.cuda.synchronize()
        ms[length] = gpu_ctx.stage_times()["seedprep"][0]
        gpu_ctx.set_timing(False)
    idx.close()
    assert ms[95_000] < 10 * ms[76_000], ms

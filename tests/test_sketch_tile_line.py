"""Reads of a tile or less at high hash ratios: both sides of the line up to which
they take the bit planes give the oracle's k-mers, and a read beyond it costs no
more than at ratio 1, where the rolling kernels have always taken it."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import xorshift_dna
from test_gpu_parity import _read_sketches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [0.26, 0.4, 0.5, 0.51, 1.0])
def test_a_tile_on_both_sides_of_the_line(r):
    for n in (int(900 / r) - 1, int(900 / r), int(900 / r) + 1, int(900 / r) + 2):
        read = xorshift_dna(n, n)
        for packed in (0, 1):
            got = _read_sketches([read], 25, r, packed)[0]
            assert all(np.array_equal(x, y) for x, y in zip(got, O.sketch(read, 25, r))), (n, packed)


def test_cost_beyond_the_line(gpu_ctx):
    import torch

    dna = np.frombuffer(xorshift_dna(9, 20_000), np.uint8)
    n = 3_800
    d = torch.zeros(n + 32, dtype=torch.uint8, device="cuda")
    d[:n] = torch.from_numpy(dna[5_000:5_000 + n].copy()).cuda()
    out, offs, ms = torch.zeros(120, dtype=torch.uint8, device="cuda"), np.array([0, n], np.int64), {}
    for r in (0.5, 1.0):
        idx = sb.SketchIndex(gpu_ctx, ["a"], dna, np.array([0, len(dna)], np.int64), 21, r)
        for rep in range(40):
            if rep == 10:
                gpu_ctx.set_timing(True)
            idx.map_reads_device(sb.Params(k=21, h_frac=r, theta=0.4), d.data_ptr(), offs, out.data_ptr())
        torch.cuda.synchronize()
        ms[r] = gpu_ctx.stage_times()["sketch"][0]
        gpu_ctx.set_timing(False)
        idx.close()
    assert ms[0.5] < 1.4 * ms[1.0], ms  # (1.8 on the planes)

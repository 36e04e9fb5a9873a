"""Windows past the ends of the sequences, where the bit planes' tiles read As: k
As can be selected (k = 26 from a hash ratio of 0.022 on), yet they are no
candidates; those of sequences of As are."""
import numpy as np
import pytest

import oracle as O
import shmap_b200 as sb

from helpers import xorshift_dna
from test_gpu_parity import _read_sketches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [20, 26])  # k As hash to 0.065 and 0.022 of the range
def test_sequences_of_as(gpu_ctx, k):
    r = 0.1
    for n in (k - 1, k, k + 1, 119 + k, 120 + k, 121 + k, 3838 + k, 3839 + k, 3840 + k, 3841 + k, 9_000):
        for seq in (b"A" * n, xorshift_dna(n, n)):
            got, want = gpu_ctx.sketch(seq, k, r), O.sketch(seq, k, r)
            assert all(len(a) == len(b) and np.array_equal(a, b) for a, b in zip(got, want)), n
    # reads side by side, the first and last of As; packed and as letters
    for ends in (k - 1, k, 200, 4_000):
        reads = [b"A" * ends, xorshift_dna(3, 77), b"A" * 61, xorshift_dna(4, 5_000), b"A" * ends]
        for packed in (0, 1):
            for lead in (0, 13):
                got = _read_sketches([xorshift_dna(5, lead)] * (lead > 0) + reads, k, r, packed)
                for a, seq in zip(got[lead > 0:], reads):
                    assert all(np.array_equal(x, y) for x, y in zip(a, O.sketch(seq, k, r))), (ends, packed, lead)


def test_cost_does_not_depend_on_k(gpu_ctx):
    """One read of 150 bases at r = 0.2: the sketch stage at the k whose As are
    selected no more than four times that at k = 25 (12 times, had they counted)."""
    import torch

    dna = np.frombuffer(xorshift_dna(9, 20_000), np.uint8)
    d = torch.zeros(182, dtype=torch.uint8, device="cuda")
    d[:150] = torch.from_numpy(dna[5_000:5_150].copy()).cuda()
    out, offs, ms = torch.zeros(120, dtype=torch.uint8, device="cuda"), np.array([0, 150], np.int64), {}
    for k in (17, 20, 25, 26, 27, 28, 31):
        idx = sb.SketchIndex(gpu_ctx, ["a"], dna, np.array([0, len(dna)], np.int64), k, 0.2)
        for rep in range(30):
            if rep == 10:
                gpu_ctx.set_timing(True)
            idx.map_reads_device(sb.Params(k=k, h_frac=0.2, theta=0.4), d.data_ptr(), offs, out.data_ptr())
        torch.cuda.synchronize()
        ms[k] = gpu_ctx.stage_times()["sketch"][0]
        gpu_ctx.set_timing(False)
        idx.close()
    assert max(ms.values()) < 4 * ms[25], ms

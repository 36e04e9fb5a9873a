"""Batches whose scratch would not fit the device: at a hash ratio of 1 a read's
k-mer, seed and probe arrays take some 85 bytes a base, so a call that fits by
its reads and bases alone does not by its scratch. It is cut smaller, with the
records of small calls; and scratch_cost (csrc/shm_map.cu) bounds what a batch
takes."""
import ctypes

import numpy as np
import pytest

import shmap_b200 as sb

from helpers import pack, record_mismatches, xorshift_dna

pytestmark = pytest.mark.gpu

READ, TIMES = 20_024, 70  # 20,000 k-mers a read: 65,536 probe slots


def test_calls_beyond_the_free_memory():
    import torch

    ref = xorshift_dna(23, 300_000)
    first = [ref[s:s + READ] for s in range(0, 250_000, 2_500)]
    p = sb.Params(k=25, h_frac=1.0, theta=0.4)
    seq1, offs1 = pack(first)
    seq = np.tile(seq1[: offs1[-1]], TIMES)  # 140 Mbases
    offs = np.arange(len(first) * TIMES + 1, dtype=np.int64) * READ
    d_seq = torch.zeros(len(seq) + 32, dtype=torch.uint8, device="cuda")
    d_seq[: len(seq)].copy_(torch.from_numpy(seq))
    d_out = torch.empty((len(offs) - 1) * sb.RECORD_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    cost = sb.lib().shm_internal_scratch_cost
    base, read = ctypes.c_double(), ctypes.c_double()
    cost(ctypes.byref(p.c()), ctypes.byref(base), ctypes.byref(read))

    def mapped(hold):
        """The records of a new context's device and host calls with `hold` bytes
        left free for them, and the bytes that it took for the device call."""
        ctx = sb.Context(0)
        idx = sb.SketchIndex.from_records(ctx, [("r", ref)], 25, 1.0)
        want = np.tile(idx.map_reads(p, seq1, offs1), TIMES)
        free = torch.cuda.mem_get_info()[0]
        rest = torch.empty(max(0, free - hold), dtype=torch.uint8, device="cuda") if hold else None
        try:
            free = torch.cuda.mem_get_info()[0]
            idx.map_reads_device(p, d_seq.data_ptr(), offs, d_out.data_ptr())
            took = free - torch.cuda.mem_get_info()[0]
            got = d_out.cpu().numpy().view(sb.RECORD_DTYPE)
            assert (want["status"] == 0).all()
            assert not record_mismatches(got, want)
            if hold:
                assert not record_mismatches(idx.map_reads(p, seq, offs), want)
        finally:
            del rest
            torch.cuda.empty_cache()
            idx.close()
            ctx.close()
        return took

    whole = mapped(0)
    bound = base.value * len(seq) + read.value * (len(offs) - 1)
    assert 9e9 < whole < bound + 1.6e9  # (and what does not grow with the batch)
    assert mapped(9_000_000_000) < 9e9

"""The device pool of temporaries and indexes keeps freed memory, up to 1 GiB,
whatever long-lived objects hold of it (csrc/shm_prims.cu)."""
import ctypes

import pytest

import shmap_b200 as sb

from helpers import xorshift_dna

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _pool(ctx):
    import torch

    torch.cuda.synchronize()  # (what is above the threshold goes back at a synchronize)
    r, u = ctypes.c_uint64(), ctypes.c_uint64()
    assert sb.lib().shm_internal_pool_bytes(ctypes.byref(r), ctypes.byref(u)) == 0
    return r.value, u.value


def test_freed_memory_is_kept_beside_objects():
    ctx = sb.Context(0)
    unit = xorshift_dna(3, 100_000)
    fasta = b">r\n" + unit * 2_000 + b"\n"  # 200 Mbases in the pool
    reserved0, used0 = _pool(ctx)
    held = [sb.DeviceFasta(ctx, fasta) for _ in range(6)]
    sb.SketchIndex.from_records(ctx, [("a", unit * 100)], 25, 0.1).close()
    reserved, used = _pool(ctx)
    assert used - used0 >= 1_200_000_000  # more than the pool keeps of freed memory
    assert 100_000_000 < reserved - used <= GIB + 64 * 2 ** 20, (reserved, used)
    for f in held:
        f.close()
    reserved, used = _pool(ctx)
    assert used <= used0 and reserved <= used + GIB + 64 * 2 ** 20, (reserved, used)
    ctx.close()

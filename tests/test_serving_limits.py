"""A server slot's batch limits (serve_limits in csrc/shm_serve.cu): batches of
any read lengths within them take no more device memory than the slot's share,
by the arrays a batch has (csrc/shm_map.cu); the longest read a request may
hold does not depend on that; shares as servers have them limit nothing."""
import ctypes
import math

import numpy as np
import pytest

import shmap_b200 as sb


def _limits(p, share, reads=16384, bases=1 << 28):
    f = sb.lib().shm_internal_serve_limits
    f.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int32, ctypes.c_int64] + [ctypes.c_void_p] * 3
    cp, r, b, m = p.c(), ctypes.c_int32(), ctypes.c_int64(), ctypes.c_int64()
    f(ctypes.byref(cp), share, reads, bases, ctypes.byref(r), ctypes.byref(b), ctypes.byref(m))
    return r.value, b.value, m.value


def _device_bytes(lens, k, r, lcs):
    """Of a batch of reads of these lengths, each buffer a quarter larger than asked for."""
    total = 0
    for n in lens:
        nw = max(0, int(n) - k + 1)
        mean = nw * r
        cap = nw if r >= 1 else min(nw, max(int(mean + 6 * math.sqrt(mean)), int(2 * mean)) + 16) if nw else 0
        slots = max(16, 1 << max(0, (2 * cap - 1).bit_length()))
        total += int(n) + cap * (8 + 4 + 4 + 16 + (8 if lcs else 0)) + 16 * slots
        total += (512 + 1024) * (24 + 4)            # bucket tables, first and spare, with their lists
        total += 64 * (88 + 3 * 4 + 2 * 40)         # jobs, their lists, the sweep's scratch
        total += sb.RECORD_DTYPE.itemsize + 19 * 4 + 4 * 8 + 28 + 5 * 8 + 16  # record, counters, plan, bins, offsets
    return 1.25 * total


@pytest.mark.parametrize("r", [0.01, 0.1, 0.45, 1.0])
@pytest.mark.parametrize("metric", ["Containment", "bucket_LCS"])
@pytest.mark.parametrize("mean", [150, 2_500, 17_000, 90_000])
def test_batches_fit_their_share(r, metric, mean):
    rng = np.random.default_rng(int(1000 * r) + mean)
    p = sb.Params(k=25, h_frac=r, theta=0.4, metric=metric)
    for share in (1 << 28, 1 << 30, 6 << 30):
        reads, bases, _ = _limits(p, share)
        lens = rng.lognormal(math.log(mean), 0.3, min(reads, max(1, int(1.2 * bases / mean)))).astype(np.int64) + 1
        lens = lens[np.cumsum(lens) <= bases]
        assert _device_bytes(lens, 25, r, metric == "bucket_LCS") <= share


def test_longest_read_and_plain_shares():
    for r in (0.01, 0.3):
        p = sb.Params(k=25, h_frac=r, theta=0.4)
        for share in (1 << 20, 1 << 28, 8 << 30):
            reads, bases, longest = _limits(p, share)
            assert longest == min(1 << 28, max(1, int(share / (1 + 128 * r))))
            assert reads >= 1 and 1 <= bases <= longest
    assert _limits(sb.Params(k=25, h_frac=0.01, theta=0.4), 8 << 30)[:2] == (16384, 1 << 28)

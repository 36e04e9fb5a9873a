"""Uploads from pageable memory through the context's pinned slots (from 64 MiB
on): sizes at the rule's line and around a multiple of a slot, and two contexts
at once from two threads, give the device the bytes that the host holds."""
import threading

import numpy as np
import pytest

import shmap_b200 as sb

pytestmark = pytest.mark.gpu
LEAST, SLOT = 64 << 20, 2 << 20


def _check(ctx, total, seed):
    rng = np.random.default_rng(seed)
    body = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 1 << 20)]
    seq = np.resize(body, total - 3)
    seq[rng.integers(0, len(seq), 4096)] = ord("N")
    data = np.concatenate([np.frombuffer(b">a\n", np.uint8), seq])
    for _ in range(2):
        fa = sb.DeviceFasta(ctx, data)
        assert fa.names == ["a"] and np.array_equal(fa.seq(), seq)
        fa.close()
        seq = seq[::-1].copy()
        data[3:] = seq


@pytest.mark.parametrize("total", [LEAST - 1, LEAST, LEAST + 1, LEAST + SLOT - 1, LEAST + SLOT, LEAST + 7 * SLOT + 5])
def test_staged_sizes(gpu_ctx, total):
    _check(gpu_ctx, total, total & 1023)


def test_two_contexts_at_once(gpu_ctx):
    ctxs = [gpu_ctx, sb.Context(0)]
    bad = []

    def run(i):
        try:
            _check(ctxs[i], LEAST + (3 + i) * SLOT + i, i)
        except BaseException as e:  # noqa: BLE001
            bad.append(e)

    th = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    ctxs[1].close()
    assert not bad, bad

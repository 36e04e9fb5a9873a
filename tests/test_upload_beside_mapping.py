"""Uploads from ordinary memory and host mapping on different contexts do not
wait for each other: an upload finishes while another thread holds the packing
of a mapping call, and mapping calls give their records beside a stream of
uploads."""
import threading

import numpy as np
import pytest

import shmap_b200 as sb

from helpers import pack, record_mismatches, xorshift_dna

pytestmark = pytest.mark.gpu


def _fasta(mib, seed):
    body = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(seed).integers(0, 4, 1 << 20)]
    return np.concatenate([np.frombuffer(b">a\n", np.uint8), np.resize(body, mib << 20)])


def _upload(ctx, data):
    fa = sb.DeviceFasta(ctx, data)
    ok = np.array_equal(fa.seq(), data[3:])
    fa.close()
    return ok


def test_upload_while_a_packing_is_held(gpu_ctx):
    hold = sb.lib().shm_internal_pack_hold
    held, release, done = threading.Event(), threading.Event(), []

    def holder():
        hold(1)
        held.set()
        release.wait(120)
        hold(0)

    h = threading.Thread(target=holder)
    h.start()
    assert held.wait(30)
    data = _fasta(96, 1)
    t = threading.Thread(target=lambda: done.append(_upload(gpu_ctx, data)))
    t.start()
    t.join(60)
    finished = not t.is_alive()
    release.set()
    h.join()
    t.join()
    assert finished and done == [True]
    assert _upload(gpu_ctx, data)  # and by its threads again


def test_mapping_beside_uploads(gpu_ctx):
    ref = xorshift_dna(3, 400_000)
    idx = sb.SketchIndex.from_records(gpu_ctx, [("r", ref)], 15, 0.05)
    seq, offs = pack([ref[s:s + 3_000] for s in range(0, 390_000, 130)])
    p = sb.Params(k=15, h_frac=0.05, theta=0.4)
    want = idx.map_reads(p, seq, offs)
    assert (want["status"] == 0).mean() > 0.9
    other, stop, ok = sb.Context(0), threading.Event(), []

    def uploads():
        data = _fasta(80, 2)
        while not stop.is_set():
            ok.append(_upload(other, data))

    t = threading.Thread(target=uploads)
    t.start()
    try:
        for _ in range(60):
            mm = record_mismatches(idx.map_reads(p, seq, offs), want)
            assert not mm, mm
    finally:
        stop.set()
        t.join()
    other.close()
    idx.close()
    assert ok and all(ok)

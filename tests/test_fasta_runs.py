"""The device parser's 64-byte runs and 16 KiB chunks: line ends, '\\r' before a
line's end, headers, blank lines and the file's end at every position around
the edges of both, against the host reader (the reference's record rules,
src/io/mod.rs:383-427). Names, offsets and bases are equal."""
import numpy as np
import pytest

import shmap_b200 as sb
from helpers import xorshift_dna
from shmap_b200 import fasta

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 62, 63, 64, 65, 127, 128, 2047, 2048, 16382, 16383, 16384, 16385, 32768]


def _same(gpu_ctx, tmp_path, data):
    p = tmp_path / "x"
    p.write_bytes(data)
    want = fasta.read_fastx(str(p))
    fa = sb.DeviceFasta(gpu_ctx, data)
    seq = fa.seq().tobytes()
    assert fa.names == [n for n, _ in want]
    assert [seq[fa.offs[i]:fa.offs[i + 1]] for i in range(fa.n)] == [s for _, s in want]
    fa.close()


@pytest.mark.parametrize("eol", [b"\n", b"\r\n", b"\r\r\n", b"\n\n", b"\r"])
def test_line_ends_at_run_and_chunk_edges(gpu_ctx, tmp_path, eol):
    for at in EDGES:
        for off in (0, 1, 2):
            body = xorshift_dna(at + off + 1, max(0, at + off - 3))
            _same(gpu_ctx, tmp_path, b">a\n" + body + eol + b"ACGT" + eol + b">b\tx" + eol + b"GG")
            _same(gpu_ctx, tmp_path, b">a\n" + body + eol)


@pytest.mark.parametrize("eol", [b"\n", b"\r\n"])
def test_fastq_lines_at_run_and_chunk_edges(gpu_ctx, tmp_path, eol):
    for at in EDGES:
        for off in (0, 1, 2):
            sq = xorshift_dna(at + off + 1, at + off)
            rec = b"@q x" + eol + sq + eol + b"+" + eol + b"@" * len(sq)
            _same(gpu_ctx, tmp_path, rec + eol + rec)
            _same(gpu_ctx, tmp_path, rec + eol * 2)


@pytest.mark.parametrize("pad", [0, 13, 16379])
def test_short_lines_and_records(gpu_ctx, tmp_path, pad):
    """Many line ends and headers inside one run."""
    rng = np.random.default_rng(pad)
    parts = [b">p\n" + b"A" * pad]
    for i in range(3000):
        parts.append([b"\n", b"\r\n", b"\nAC", b"\n>", b"\n>r%d" % i, b"G\r", b">", b" "][int(rng.integers(0, 8))])
    _same(gpu_ctx, tmp_path, b"".join(parts))

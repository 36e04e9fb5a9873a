"""bucket_LCS where the longest read's position bitmap fills the 48 KiB of
shared memory that a kernel has without asking for more: a process whose first
such call is of that size (what one kernel asked for outlives a context)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUN = """
import sys
for p in ("shmap-rs_b200", "oracle", "tests"): sys.path.insert(0, p)
import numpy as np, oracle as O, shmap_b200 as sb
from helpers import pack, record_mismatches
n, rng = int(sys.argv[1]), np.random.default_rng(1)
dna = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n + 40_000)].tobytes()
read = bytearray(dna[20_000:20_000 + n])
for i in range(500, n, 997): read[i] = 65
seq, offs = pack([bytes(read), dna[1_000:9_000]])
ref = [("a", dna)]
kw = dict(k=15, h_frac=0.01, theta=0.4, metric="bucket_LCS")
g, o = sb.SketchIndex.from_records(sb.Context(0), ref, 15, 0.01), O.Index.from_records(ref, 15, 0.01)
rec = g.map_reads(sb.Params(**kw), seq, offs)
assert not record_mismatches(rec, o.map_reads(O.params(**kw), seq, offs)), "records differ"
assert (rec["status"] == 0).all()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("bases", [261_400, 261_500, 262_143, 262_144, 262_145, 393_216, 393_217])
def test_first_call(bases):
    p = subprocess.run([sys.executable, "-c", RUN, str(bases)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-800:]

"""The device-buffer calls under stream capture when the captured call is the
process's first of its size.  Everything that a launch needs is loaded and set
up when the filter is created, so that the call only records its launches."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys, time
sys.path.insert(0, sys.argv[1])
n = int(sys.argv[2])
import numpy as np
import torch
import cusbf_b200 as sbf
from oracle import oracle
cfg = dict(k=31, s=28, m=16, hashes=int(sys.argv[3]))
rng = np.random.default_rng(n)
seq = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)]
f = sbf.Filter(1 << 20, **cfg)
d = torch.from_numpy(seq.copy()).cuda()
out = torch.full((n - 30,), 7, dtype=torch.uint8, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    st = torch.cuda.current_stream().cuda_stream
    t = [time.perf_counter()]
    f.insert_sequence_async(d[:n // 2], stream=st)
    t.append(time.perf_counter())
    f.contains_sequence_async(d, out, stream=st)
    t.append(time.perf_counter())
g.replay()
torch.cuda.synchronize()
o = oracle.Oracle(**cfg)
w = o.new_words(1 << 20)
o.insert(w, seq[:n // 2])
assert (f.words_host() == w).all()
assert (out.cpu().numpy() == o.contains(w, seq)).all()
print("insert %.0f query %.0f us" % tuple((b - a) * 1e6 for a, b in zip(t, t[1:])))
"""


@pytest.mark.parametrize("n,hashes", [(5_000, 4), (1_000_000, 4), (1_000_000, 16)])
def test_first_call_under_capture(cuda, oracle_mod, n, hashes):
    """Right results, and the first call within 2 ms on the host (recording a
    launch takes about 0.1 ms, loading its kernel took 4)."""
    def first_call():
        r = subprocess.run([sys.executable, "-c", CODE, ROOT, str(n), str(hashes)],
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return float(r.stdout.split()[1])

    # Other processes can hold the host up: the better of three.
    assert min(first_call() for _ in range(3)) < 2_000

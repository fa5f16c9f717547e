"""First transforms of lines of different lengths from many threads at once
(GPU): one kernel serves every length and each length wants its own amount of
shared memory.  In a process of its own, where nothing has been launched yet.
"""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import threading
import numpy as np
import torch
from dftpy_gb300 import _lib
L = _lib.load()
lengths = [n for n in range(180, 900) if all(n % p for p in (11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47))
           and max(p for p in range(2, n + 1) if n % p == 0 and all(p % q for q in range(2, p))) <= 7][::3]
gate = threading.Barrier(len(lengths))
bad = []
def run(n):
    try:
        nr = [6, n, 8]
        plan = _lib.Plan(nr, np.diag([1.0 * k for k in nr]), precision=1)
        x = np.random.default_rng(n).standard_normal(nr)
        xd = torch.tensor(x, device="cuda")
        out = torch.empty((6, n, 5), dtype=torch.complex128, device="cuda")
        with torch.cuda.stream(torch.cuda.Stream()):
            gate.wait(60)
            _lib.check(L.gbofdft_fft_r2c(plan.handle, _lib.ptr(xd), _lib.ptr(out), _lib.stream_ptr()))
            torch.cuda.current_stream().synchronize()
        ref = np.fft.rfftn(x)
        if not np.abs(out.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max():
            bad.append((n, "wrong"))
    except Exception as e:
        bad.append((n, repr(e)))
torch.zeros(1, device="cuda")
ts = [threading.Thread(target=run, args=(n,)) for n in lengths]
[t.start() for t in ts]
[t.join() for t in ts]
print(bad)
raise SystemExit(1 if bad else 0)
"""


def test_lengths_from_threads():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

"""The radial tables' spline where the library is not built: the same coefficients.

Tolerance: both eliminate the same diagonally dominant system, whose inverse
amplifies an error below 1 for spacings that differ by less than 4; a few dozen
roundings of the largest coefficient."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [4, 5, 6, 33, 1000])
def test_spline_without_library(n, tmp_path):
    from dftpy_gb300._tables import spline_notaknot
    rng = np.random.default_rng(n)
    x, y = np.cumsum(rng.uniform(0.25, 1.0, n)), rng.standard_normal(n)
    np.savez(tmp_path / "in.npz", x=x, y=y)
    code = ("import numpy as np\nfrom dftpy_gb300._tables import spline_notaknot\nd = np.load('in.npz')\n"
            "np.savez('out.npz', c=spline_notaknot(d['x'], d['y'])[1])\n")
    env = dict(os.environ, GBOFDFT_LIBRARY=str(tmp_path / "none.so"),
               PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    subprocess.run([sys.executable, "-c", code], cwd=tmp_path, env=env, check=True, timeout=300)
    c = spline_notaknot(x, y)[1]
    got = np.load(tmp_path / "out.npz")["c"]
    assert got.shape == c.shape
    np.testing.assert_allclose(got, c, rtol=0, atol=256 * 2.0 ** -53 * np.abs(c).max())


def test_spline_that_does_not_fit_in_memory():
    """A status, no exception through the C entry (which would end the process)."""
    code = ("import ctypes\nfrom dftpy_gb300 import _lib\nx = (ctypes.c_double * 4)(0, 1, 2, 3)\n"
            "p = ctypes.cast(x, ctypes.c_void_p)\nrc = _lib.load().gbofdft_spline(1 << 60, p, p, p)\n"
            "assert rc == 4 and 'memory' in _lib.last_error(), rc\n")
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr

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

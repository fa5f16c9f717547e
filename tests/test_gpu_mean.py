"""gbofdft_mean (GPU): ends before and after the 16-byte loads, fewer values
than threads, more than one round of the grid.  The sum is exact to FP64
rounding: |error| <= 64 eps sum|x| / n for at most 64 additions in a chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("off", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 255, 1025, 622593, 4000001])
def test_mean(n, off, dtype):
    import torch
    from dftpy_gb300 import _lib
    _lib.require_cuda()
    x = np.random.default_rng(n).standard_normal(n + off).astype(dtype)
    xd = torch.tensor(x, device="cuda")[off:]
    want = np.longdouble(x[off:]).sum() / n
    bound = 64 * 2.0 ** -53 * np.abs(x[off:]).astype(np.float64).sum() / n
    assert abs(_lib.mean(xd) - float(want)) <= bound


def test_mean_values_and_refusals():
    import torch
    from dftpy_gb300 import _lib
    _lib.require_cuda()
    x = torch.ones((4, 5, 6), device="cuda", dtype=torch.float64)
    assert _lib.mean(x.permute(2, 0, 1)) == 1.0
    x[1, 2, 3] = float("inf")
    assert _lib.mean(x) == float("inf")
    x[0, 0, 0] = float("nan")
    assert np.isnan(_lib.mean(x))
    assert _lib.mean(torch.ones(7, device="cuda", dtype=torch.float16)) == 1.0
    with pytest.raises(ValueError):
        _lib.mean(torch.ones(3, dtype=torch.float64))

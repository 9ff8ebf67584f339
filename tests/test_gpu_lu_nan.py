"""Pivots of systems that hold NaN: any number is taken before a NaN, so a column
of zeros and NaN has a zero pivot, whatever the size of the system."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ttnumpy_b200 import kernels

    return kernels


def solve(K, a, b):
    cols = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    x = torch.from_numpy(b.copy()).cuda()
    info = torch.full((1,), -9, dtype=torch.int32, device="cuda")
    K.lu_solve_(cols, x, info)
    return int(info.item()), x.cpu().numpy()


@pytest.mark.parametrize("n", [2, 33, 100, 160, 161, 300, 1030])
@pytest.mark.parametrize("at", [0, 1])
def test_zero_pivot_beside_a_nan(K, n, at):
    """Column 0 is zero but for one NaN: LAPACK's search, which compares numbers
    and skips NaN, finds the zero pivot."""
    a = np.random.default_rng(n).standard_normal((n, n))
    a[:, 0] = 0.0
    a[at, 0] = np.nan
    assert solve(K, a, np.ones(n))[0] == 1


@pytest.mark.parametrize("n", [2, 33, 100, 160, 161, 300])
def test_nan_beside_numbers(K, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a[n // 2, 0] = np.nan
    info, x = solve(K, a, np.ones(n))
    assert info == 0 and np.isnan(x).all()


@pytest.mark.parametrize("n", [1030, 1700])
def test_column_of_nan(K, n):
    """Beyond the registers: once only rows of NaN are left, a column has no
    largest entry; its pivot stays on the diagonal."""
    a = np.random.default_rng(n).standard_normal((n, n))
    a[n // 2, 0] = np.nan
    info, x = solve(K, a, np.ones(n))
    assert info == 0 and np.isnan(x).all()
    a[:] = np.nan
    info, x = solve(K, a, np.ones(n))
    assert info == 0 and np.isnan(x).all()

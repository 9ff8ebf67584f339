"""The TTM-by-TT product core at the edges of its blocks: ragged columns and
rows, several column modes, modes too large for shared memory, and infinities
and NaN, which spread through the operator's zeros as in the dense product.
"""

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


def product(K, op, core):
    got = K.kron(torch.from_numpy(op).cuda(), torch.from_numpy(core).cuda())
    with np.errstate(invalid="ignore"):
        want = np.einsum("aijb,xjky->axikby", op, core).reshape(got.shape)
    return got.cpu().numpy(), want


def banded(rng, ra, n, m, ra2):
    op = rng.standard_normal((ra, n, m, ra2))
    return op * (np.abs(np.arange(n)[:, None] - np.arange(m)) < 2)[None, :, :, None]


@pytest.mark.parametrize("ra,n,m,ra2,rx,kk,rx2", [(1, 1, 1, 1, 1, 1, 1), (6, 2, 2, 6, 8, 1, 8),
                                                  (4, 33, 31, 3, 5, 1, 7), (2, 64, 64, 4, 3, 1, 129),
                                                  (3, 5, 70, 2, 4, 3, 45), (2, 3, 900, 2, 2, 1, 40),
                                                  (1, 40, 257, 1, 2, 2, 33)])
@pytest.mark.parametrize("dense", [False, True])
def test_kron_edges(K, ra, n, m, ra2, rx, kk, rx2, dense):
    rng = np.random.default_rng(ra * n + m + rx2)
    op = rng.standard_normal((ra, n, m, ra2)) if dense else banded(rng, ra, n, m, ra2)
    core = rng.standard_normal((rx, m, kk, rx2))
    got, want = product(K, op, core)
    assert np.linalg.norm(got - want) <= 1e-14 * np.linalg.norm(want)


def test_kron_spreads_non_finite_values(K):
    rng = np.random.default_rng(1)
    op = banded(rng, 2, 9, 9, 2)
    core = rng.standard_normal((3, 9, 1, 5))
    core[1, 4, 0, 2] = np.inf
    core[2, 0, 0, 1] = np.nan
    got, want = product(K, op, core)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    fine = np.isfinite(want)
    assert np.abs(got[fine] - want[fine]).max() < 1e-13

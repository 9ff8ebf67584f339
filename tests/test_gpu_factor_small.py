"""SVDs of few columns, which are iterated on without pivoted QRs, up to the
width where those begin: full and deficient rank, steep spectra, zeros, either
factor alone, wide and tall."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ttnumpy_b200 import kernels

    return kernels


def matrix(kind, m, k):
    rng = np.random.default_rng(100 * m + k)
    a = rng.standard_normal((m, k))
    if kind == "steep":
        a = a @ np.diag(10.0 ** -np.arange(0, 3 * k, 3))
    elif kind == "deficient":
        a[:, -1] = a[:, 0]
    elif kind == "zero column":
        a[:, k // 2] = 0.0
    elif kind == "zero":
        a[:] = 0.0
    return a


@pytest.mark.parametrize("k", [1, 2, 3, 6, 7])
@pytest.mark.parametrize("m", [7, 300, 9001])
def test_small_svd(K, m, k):
    for kind in ("full", "steep", "deficient", "zero column", "zero"):
        for wide in (False, True):
            a = matrix(kind, m, k)
            check(K, a.T if wide else a, m, k)


def check(K, a, m, k):
    dev = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    u, s, vh = (x.cpu().numpy() for x in K.svd(dev))
    # a QR with sums of m / 32 terms a lane, then at most 60 sweeps of rotations,
    # each column rotated k - 1 times a sweep; convergence takes about 6
    tol = 4 * k * (m / 32 + 16 + 6 * k) * EPS
    norm = np.linalg.norm(a) or 1.0
    assert np.linalg.norm((u * s) @ vh - a) <= tol * norm
    assert np.linalg.norm(u.T @ u - np.eye(k)) <= tol
    assert np.linalg.norm(vh @ vh.T - np.eye(k)) <= tol
    assert (np.diff(s) <= 0).all()
    assert np.abs(s - np.linalg.svd(a, compute_uv=False)).max() <= tol * norm
    u1, s1, none = K.svd(dev, want_vh=False)
    assert none is None
    u1, s1 = u1.cpu().numpy(), s1.cpu().numpy()
    assert np.linalg.norm(u1.T @ u1 - np.eye(k)) <= tol and np.abs(s1 - s).max() <= tol * norm
    assert np.linalg.norm(u1 @ (u1.T @ a) - a) <= tol * norm
    none, s2, v2 = K.svd(dev, want_u=False)
    assert none is None
    v2, s2 = v2.cpu().numpy(), s2.cpu().numpy()
    assert np.linalg.norm(v2 @ v2.T - np.eye(k)) <= tol and np.abs(s2 - s).max() <= tol * norm
    assert np.linalg.norm((a @ v2.T) @ v2 - a) <= tol * norm


def test_small_svd_of_nan_ends(K):
    a = torch.full((20, 3), float("nan"), dtype=torch.float64, device="cuda")
    u, s, vh = K.svd(a)
    assert torch.isnan(s).all() and u.shape == (20, 3) and vh.shape == (3, 3)


@pytest.mark.parametrize("k", [1, 3, 6, 8])
def test_a_nan_leaves_no_singular_value(K, k):
    a = np.random.default_rng(k).standard_normal((40, k))
    a[7, k // 2] = np.nan
    u, s, vh = K.svd(torch.from_numpy(a).cuda())
    assert torch.isnan(s).all() and torch.isnan(vh).all() and torch.isnan(u).any()

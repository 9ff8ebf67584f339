"""The limits that the header states for the QR and SVD entry points: what fits
shared memory, and what ttb_qr_static takes.  Each refusal is the host's."""

import ctypes as C

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


def factor(K, name, a, work=None):
    from ttnumpy_b200 import _lib

    m, k = a.shape
    p = min(m, k)
    dev = torch.from_numpy(a).cuda()
    q, r = K.empty(m, p), K.empty(p, k)
    d = (_lib.QR * 1)(_lib.QR(K.ptr(dev), k, 1, K.ptr(q), p, 1, K.ptr(r), k, 1, K.ptr(work), m, k))
    code = getattr(K.lib(), name)(d, 1, K.stream())
    torch.cuda.synchronize()
    return code, q.cpu().numpy(), r.cpu().numpy()


def check(a, q, r):
    m, k = a.shape
    tol = 4 * k * (m / 32 + 16) * EPS  # k reflectors, sums of m / 32 terms a lane, twice
    assert np.linalg.norm(q @ r - a) <= tol * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(q.shape[1])) <= tol


@pytest.mark.parametrize("m,k", [(160, 159), (200, 127), (1448, 1447)])
def test_static_takes_what_the_header_says(K, m, k):
    """8 (m k + min(m, k)) bytes up to 200 KiB in shared memory, beyond that m k +
    min(m, k) doubles of the array's 2^21, each just within its limit."""
    a = np.random.default_rng(m).standard_normal((m, k))
    code, q, r = factor(K, "ttb_qr_static", a)
    assert code == 0
    check(a, q, r)


def test_static_refuses_more(K):
    a = np.random.default_rng(0).standard_normal((1449, 1448))
    assert factor(K, "ttb_qr_static", a)[0] == -2


@pytest.mark.parametrize("m,k", [(600, 8), (600, 40), (1600, 15), (3000, 8), (160, 159)])
def test_qr_without_work_areas_in_shared_memory(K, m, k):
    a = np.random.default_rng(m).standard_normal((m, k))
    code, q, r = factor(K, "ttb_qr", a)
    assert code == 0
    check(a, q, r)


def svd(K, a):
    from ttnumpy_b200 import _lib

    m, k = a.shape
    dev = torch.from_numpy(a).cuda()
    u, s, vh = K.empty(m, k), K.empty(k), K.empty(k, k)
    d = (_lib.SVD * 1)(_lib.SVD(K.ptr(dev), k, 1, K.ptr(u), k, 1, K.ptr(s), K.ptr(vh), k, 1, None,
                                None, m, k))
    code = K.lib().ttb_svd(d, 1, K.stream())
    torch.cuda.synchronize()
    return code, u.cpu().numpy(), s.cpu().numpy(), vh.cpu().numpy()


@pytest.mark.parametrize("m,k", [(700, 20), (2000, 10)])
def test_svd_without_work_areas_in_shared_memory(K, m, k):
    a = np.random.default_rng(m).standard_normal((m, k))
    code, u, s, vh = svd(K, a)
    assert code == 0
    tol = (4 * k * (m / 32 + 16) + 24 * k * k) * EPS  # the QR, and six sweeps of rotations
    assert np.linalg.norm((u * s) @ vh - a) <= tol * np.linalg.norm(a)


def test_what_does_not_fit_is_refused_without_work_areas(K):
    before = K.launch_count()
    a = np.random.default_rng(0).standard_normal((900, 40))
    assert factor(K, "ttb_qr", a)[0] == 1  # cudaErrorInvalidValue
    assert svd(K, a)[0] == 1
    assert K.launch_count() == before

"""Tall matrices that one block factors sooner than a tree of row blocks take one
launch, the others several; both are right on either side of the lines."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
EPS = np.finfo(float).eps
BLOCK = [(513, 1), (8192, 1), (2730, 3), (2048, 8), (1024, 16), (768, 32), (521, 49)]
TREE = [(8193, 1), (2731, 3), (2049, 8), (1025, 9), (1025, 16), (900, 32), (640, 48)]


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ttnumpy_b200 import kernels

    return kernels


def launches(K, f):
    before = K.launch_count()
    out = f()
    return out, K.launch_count() - before


def bound(m, k):
    return 4 * k * (m / 32 + 16) * EPS  # k reflectors, sums of m / 32 terms a lane, twice


@pytest.mark.parametrize("m,k", BLOCK + TREE)
def test_qr_route(K, m, k):
    a = np.random.default_rng(m).standard_normal((m, k))
    (q, r), n = launches(K, lambda: K.qr(torch.from_numpy(a).cuda()))
    assert (n == 1) == ((m, k) in BLOCK)
    q, r = q.cpu().numpy(), r.cpu().numpy()
    assert np.linalg.norm(q @ r - a) <= bound(m, k) * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(k)) <= bound(m, k)
    assert np.array_equal(np.sign(np.diag(r)), np.sign(np.diag(np.linalg.qr(a)[1])))


@pytest.mark.parametrize("m,k,block", [(16384, 1, True), (4096, 4, True), (16385, 1, False),
                                       (1639, 10, False), (1024, 16, True), (1024, 24, True)])
def test_r_route(K, m, k, block):
    a = np.random.default_rng(m).standard_normal((m, k))
    (_, r), n = launches(K, lambda: K.qr(torch.from_numpy(a).cuda(), want_q=False))
    assert (n == 1) == block
    want = np.linalg.qr(a)[1]
    assert np.linalg.norm(r.cpu().numpy() - want) <= bound(m, k) * np.linalg.norm(a)


@pytest.mark.parametrize("m,k,block", [(6144, 1, True), (2048, 3, True), (1024, 16, True),
                                       (6145, 1, False), (1024, 17, False), (1025, 16, False)])
def test_svd_route(K, m, k, block):
    a = np.random.default_rng(m).standard_normal((m, k))
    (u, s, vh), n = launches(K, lambda: K.svd(torch.from_numpy(a).cuda()))
    assert (n == 1) == block
    u, s, vh = (x.cpu().numpy() for x in (u, s, vh))
    tol = bound(m, k) + 24 * k * k * EPS  # and some six sweeps of k - 1 rotations a column
    assert np.linalg.norm((u * s) @ vh - a) <= tol * np.linalg.norm(a)
    assert np.linalg.norm(u.T @ u - np.eye(k)) <= tol
    assert np.linalg.norm(vh @ vh.T - np.eye(k)) <= tol

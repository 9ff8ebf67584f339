"""QR of narrow matrices, which are factored column by column in one block, at
the widths and heights where the form changes."""

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


def bound(m, k):
    # a reflector's sums run over m / 32 terms a lane and a tree of 16; k of
    # them, twice with Q, each of two operations a term
    return 4 * k * (m / 32 + 16) * EPS


@pytest.mark.parametrize("k", [1, 2, 4, 5])
@pytest.mark.parametrize("m", [5, 33, 34, 129, 130, 257, 513, 2048, 2049, 5001])
@pytest.mark.parametrize("flip", [False, True])
def test_narrow_qr(K, m, k, flip):
    rng = np.random.default_rng(m + k)
    a = rng.standard_normal((m, k))
    dev = torch.from_numpy(a.T.copy()).cuda().t() if flip else torch.from_numpy(a).cuda()
    q, r = (x.cpu().numpy() for x in K.qr(dev))
    lq, lr = np.linalg.qr(a)
    assert np.linalg.norm(q @ r - a) <= bound(m, k) * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(k)) <= bound(m, k)
    assert np.array_equal(np.sign(np.diag(r)), np.sign(np.diag(lr)))
    assert np.array_equal(np.tril(r, -1), np.zeros((k, k)))
    _, r1 = K.qr(dev, want_q=False)
    assert np.linalg.norm(r1.cpu().numpy() - r) <= bound(m, k) * np.linalg.norm(a)


def test_narrow_qr_of_a_zero_column(K):
    a = np.random.default_rng(1).standard_normal((300, 3))
    a[:, 1] = 0.0
    q, r = (x.cpu().numpy() for x in K.qr(torch.from_numpy(a).cuda()))
    assert np.linalg.norm(q @ r - a) <= bound(300, 3) * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(3)) <= bound(300, 3)

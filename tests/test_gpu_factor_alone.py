"""A factorisation's bits do not depend on the other problems of its call."""

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


def matrices():
    rng = np.random.default_rng(0)
    shapes = [(700, 48), (30, 7), (1500, 20), (513, 96), (2100, 3)] + [(900, 33)] * 18
    return [torch.from_numpy(rng.standard_normal(s)).cuda() for s in shapes]


@pytest.mark.parametrize("want_q", [True, False])
def test_qr_alone_equals_grouped(K, want_q):
    """Twenty-one tall problems and a small one in one call."""
    mats = matrices()
    for a, (q, r) in list(zip(mats, K.qr_many([(a, want_q, True, None, None) for a in mats])))[:6]:
        q1, r1 = K.qr(a, want_q=want_q)
        assert torch.equal(r, r1)
        assert not want_q or torch.equal(q, q1)


def test_svd_alone_equals_grouped(K):
    mats = matrices() + [a.t() for a in matrices()[:2]]
    got = K.svd_many(mats)
    for i in (0, 1, 2, 3, 4, 5, len(mats) - 2, len(mats) - 1):
        for x, y in zip(got[i], K.svd(mats[i])):
            assert torch.equal(x, y)

"""The factorisation kernels at the edges of their register tiles, against
LAPACK (SciPy).

A Householder column belongs to 8, 16 or 32 lanes by the number of rows, the
Jacobi iteration and its preconditioners come in tiles of 16 to 256 columns.
Tolerances are those of the other factorisation tests: reconstruction and
singular values to 1e-13 of the matrix, orthonormality to 1e-12.
"""

import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ttnumpy_b200 import kernels

    return kernels


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def orth(q):
    return np.abs(q.T @ q - np.eye(q.shape[1])).max()


@pytest.mark.parametrize("m", [31, 33, 64, 65, 129, 256, 257, 513, 1024, 1025, 2048, 2049])
@pytest.mark.parametrize("k", [1, 15, 66])
def test_qr_tile_edges(K, m, k):
    rng = np.random.default_rng(m + k)
    a = rng.standard_normal((m, k))
    q, r = (t.cpu().numpy() for t in K.qr(dev(a)))
    r_ref = sla.qr(a, mode="r")[0][: min(m, k)]
    assert np.linalg.norm(q @ r - a) < 1e-13 * np.linalg.norm(a)
    assert orth(q) < 1e-13
    assert np.linalg.norm(r - r_ref) < 1e-11 * np.linalg.norm(r_ref)


@pytest.mark.parametrize("m,k", [(1, 1), (9, 8), (16, 17), (33, 32), (64, 65), (97, 96),
                                 (130, 128), (129, 129), (40, 257), (260, 257), (600, 20),
                                 (20, 3000), (100, 300), (193, 200), (390, 385), (513, 512),
                                 (520, 514)])
@pytest.mark.parametrize("deficient", [False, True])
def test_svd_one_factor(K, m, k, deficient):
    """Both factors, the left one alone and the right one alone agree with
    LAPACK, also where singular values are exactly zero (equal and zero
    columns): every factor asked for is orthonormal."""
    rng = np.random.default_rng(m * k + deficient)
    p = min(m, k)
    a = rng.standard_normal((m, k)) * np.logspace(0, -8, k)
    if deficient:
        a[:, k // 2:] = 0.0
        a[m // 2:] = 0.0
    x = dev(a)
    s_ref = sla.svdvals(a)
    scale = max(np.linalg.norm(a), 1e-300)
    u, s, vh = (t.cpu().numpy() for t in K.svd(x))
    assert np.linalg.norm((u * s) @ vh - a) < 1e-13 * scale
    ul, sl, none = K.svd(x, want_vh=False)
    assert none is None
    none, sr, vr = K.svd(x, want_u=False)
    assert none is None
    for got in (s, sl.cpu().numpy(), sr.cpu().numpy()):
        assert np.abs(got - s_ref).max() <= 1e-13 * scale
    ul, vr = ul.cpu().numpy(), vr.cpu().numpy()
    for factor in (u, ul, vh.T, vr.T):
        assert factor.shape[1] == p
        assert orth(factor) < 1e-12
    assert np.linalg.norm(ul @ (ul.T @ a) - a) < 1e-12 * scale
    assert np.linalg.norm((a @ vr.T) @ vr - a) < 1e-12 * scale


@pytest.mark.parametrize("n", [2, 32, 33, 65, 97, 129, 160, 161, 177, 257, 530, 1024, 1025])
def test_lu_tile_edges(K, n):
    """Whole systems in registers up to 160 unknowns, 16-column panels with
    128-column strips beyond, row by row past 1024: against LAPACK, with rows
    that need swapping and exact ties in the pivot search."""
    rng = np.random.default_rng(n)
    a = rng.integers(-2, 3, (n, n)).astype(float) + n * 0.1 * np.eye(n)[rng.permutation(n)]
    b = rng.standard_normal(n)
    x = dev(b)
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    K.lu_solve_(dev(a.T), x, info)
    assert info.item() == 0
    want = np.linalg.solve(a, b)
    bound = 1e-13 * max(1.0, np.linalg.cond(a))
    assert np.linalg.norm(x.cpu().numpy() - want) < bound * np.linalg.norm(want)


@pytest.mark.parametrize("n,at", [(40, 40), (150, 7), (300, 1), (300, 290), (600, 333)])
def test_lu_zero_pivot(K, n, at):
    """The first exactly-zero pivot is reported by its 1-based index."""
    a = np.triu(np.ones((n, n)))
    a[at - 1, at - 1] = 0.0
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    K.lu_solve_(dev(a.T), dev(np.ones(n)), info)
    assert info.item() == at


@pytest.mark.parametrize("m,k", [(511, 30), (512, 96), (513, 97), (600, 128), (769, 2), (1025, 64),
                                 (2305, 33), (5000, 128), (20000, 5)])
def test_tall_trees(K, m, k):
    """Tall matrices go as trees of row blocks (from 512 rows, up to 128
    columns; short last nodes, odd heights): LAPACK's R with its signs, with
    and without Q, from row- and column-major storage, and several in one
    call."""
    rng = np.random.default_rng(m + k)
    a = rng.standard_normal((m, k)) * np.logspace(0, -6, k)
    r_ref = sla.qr(a, mode="r")[0][:k]
    x = dev(a)
    both = K.qr_many([(x, True, True, None, None), (dev(a.T).t(), True, True, None, None),
                      (x, False, True, None, None), (x[:40], True, True, None, None)])
    for q, r in both[:3]:
        r = r.cpu().numpy()
        assert np.linalg.norm(r - r_ref) < 1e-11 * np.linalg.norm(r_ref)
        if q is not None:
            q = q.cpu().numpy()
            assert np.linalg.norm(q @ r - a) < 1e-13 * np.linalg.norm(a)
            assert orth(q) < 1e-13
    u, s, vh = (t.cpu().numpy() for t in K.svd(x.t()))
    assert np.abs(s - sla.svdvals(a)).max() <= 1e-13 * s[0]
    assert np.linalg.norm((u * s) @ vh - a.T) < 1e-13 * np.linalg.norm(a)
    assert orth(u) < 1e-12 and orth(vh.T) < 1e-12
    for want in ({"want_u": False}, {"want_vh": False}):
        u, s1, vh = K.svd(x, **want)
        factor = (u if u is not None else vh.t()).cpu().numpy()
        assert orth(factor) < 1e-12
        assert np.abs(s1.cpu().numpy() - s).max() <= 1e-13 * s[0]

"""The forms of the TTM-by-TT product core at their limits: outputs one by one,
rows of outputs to a warp, and operator rows searched for their nonzeros, with
dense rows, ragged modes and columns, few rows and modes beyond shared memory.
Every form adds the same terms in the same order."""

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


def operator(rng, ra, n, m, ra2, dense):
    op = rng.standard_normal((ra, n, m, ra2))
    if not dense:
        op *= (np.abs(np.arange(n)[:, None] - np.arange(m)) < 2)[None, :, :, None]
    return op


def run(K, op, core):
    return K.kron(torch.from_numpy(op).cuda(), torch.from_numpy(core).cuda()).cpu().numpy()


SHAPES = [
    (64, 2, 2, 64, 1, 1, 1), (5, 3, 15, 4, 9, 2, 11),                    # one by one
    (12, 20, 3, 7, 10, 1, 5), (3, 40, 15, 33, 10, 2, 1),                 # a warp a row
    (1, 8, 16, 2, 5, 1, 7), (9, 16, 16, 9, 12, 1, 10),                   # mode 16: few, many outputs
    (1, 1, 32, 1, 1, 1, 1), (3, 7, 33, 5, 2, 1, 31), (2, 70, 64, 3, 3, 1, 65),
    (2, 65, 96, 1, 2, 3, 43), (1, 300, 257, 1, 2, 1, 9), (1, 19, 801, 2, 2, 1, 33),
]


@pytest.mark.parametrize("ra,n,m,ra2,rx,kk,rx2", SHAPES)
@pytest.mark.parametrize("dense", [False, True])
def test_forms_match_the_dense_product(K, ra, n, m, ra2, rx, kk, rx2, dense):
    rng = np.random.default_rng(n * m + rx2)
    op = operator(rng, ra, n, m, ra2, dense)
    core = rng.standard_normal((rx, m, kk, rx2))
    got = run(K, op, core)
    want = np.einsum("aijb,xjky->axikby", op, core).reshape(got.shape)
    # m terms an output, each rounded once: m eps of the sum of magnitudes
    most = np.einsum("aijb,xjky->axikby", np.abs(op), np.abs(core)).reshape(got.shape)
    assert (np.abs(got - want) <= 2 * m * np.finfo(float).eps * most).all()


@pytest.mark.parametrize("dense", [False, True])
def test_forms_give_the_same_bits(K, dense):
    """A mode-16 product large enough to be searched, against its slices, which
    are formed output by output."""
    rng = np.random.default_rng(3)
    op = operator(rng, 4, 16, 16, 4, dense)
    core = rng.standard_normal((40, 16, 1, 40))
    whole = run(K, op, core).reshape(4, 40, 16, 1, 4, 40)
    for x in (0, 17, 39):
        part = run(K, op, core[x:x + 1]).reshape(4, 1, 16, 1, 4, 40)
        assert np.array_equal(part[:, 0], whole[:, x])


@pytest.mark.parametrize("ra,n,m,ra2,rx,kk,rx2", [SHAPES[0], SHAPES[2], SHAPES[7], SHAPES[11]])
def test_forms_spread_non_finite_values(K, ra, n, m, ra2, rx, kk, rx2):
    rng = np.random.default_rng(5)
    op = operator(rng, ra, n, m, ra2, False)
    core = rng.standard_normal((rx, m, kk, rx2))
    core[0, m // 2, 0, 0] = np.inf
    core[-1, 0, 0, -1] = np.nan
    got = run(K, op, core)
    with np.errstate(invalid="ignore"):
        want = np.einsum("aijb,xjky->axikby", op, core).reshape(got.shape)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))

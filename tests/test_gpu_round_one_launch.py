"""Rounding a small train in one launch against the core-by-core sweeps (the
general path) and the oracle: the largest and smallest trains that fit, trains
just beyond, TTM trains, strided cores, caps and zero trains.
"""

import numpy as np
import pytest

from oracle import tt_oracle as O
from ttnumpy_b200 import problems as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def tt():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ttnumpy_b200

    return ttnumpy_b200


def sweeps(t, error, max_rank):
    """The general path: a QR sweep, then the SVD sweep."""
    return t.orthonormalize(canonical="left").compress_svd(error, max_rank)


def diff(a, b):
    a, b = O.Train(a.to_numpy()), O.Train(b.to_numpy())
    return O.tt_norm(O.add(a, O.scale(b, -1.0))) / max(O.tt_norm(b), 1e-300)


@pytest.mark.parametrize("d,n,r,fits", [(2, 1, 1, True), (2, 256, 1, True), (2, 257, 1, False),
                                        (5, 4, 64, True), (5, 4, 65, False), (4, 5, 52, False),
                                        (64, 2, 3, True), (65, 2, 3, False), (9, 3, 17, True)])
@pytest.mark.parametrize("error,max_rank", [(1e-6, None), (0.0, 4)])
def test_matches_general_path(tt, d, n, r, fits, error, max_rank):
    from ttnumpy_b200.tensor_train import round_in_one_launch

    t = tt.TensorTrain(P.random_tt([n] * d, r, seed=d + r))
    before = t.to_numpy()
    assert (round_in_one_launch(t.cores, error, max_rank) is not None) == fits
    got, want = t.truncate(error=error, max_rank=max_rank), sweeps(t, error, max_rank)
    assert got.bonds == want.bonds and got.orth_center == want.orth_center == 0
    assert diff(got, want) < 1e-12
    for c in got.cores[1:]:
        m = c.reshape(c.shape[0], -1).cpu().numpy()
        assert np.abs(m @ m.T - np.eye(m.shape[0])).max() < 1e-12
    assert all(np.array_equal(a, b) for a, b in zip(before, t.to_numpy()))


def test_operator_strided_and_inplace(tt):
    A = tt.TensorTrain(P.laplacian_nd(5, 4))
    got = A.truncate(error=1e-12)
    assert got.is_ttm() and got.physical_dims() == A.physical_dims()
    assert diff(got, sweeps(A, 1e-12, None)) < 1e-12
    t = tt.TensorTrain(P.random_tt([3] * 6, 5, seed=1))
    u = tt.TensorTrain._wrap([c.permute(3, 1, 2, 0).contiguous().permute(3, 1, 2, 0)
                              for c in t.cores])
    assert diff(u.truncate(error=1e-9), t.truncate(error=1e-9)) < 1e-12
    cores = t.cores
    assert t.truncate(error=1e-3, inplace=True) is t and t.cores is cores


def test_zero_train_and_errors(tt):
    z = tt.zeros([3, 4, 5], ranks=4).truncate(error=1e-6)
    assert z.bonds == [1, 1, 1, 1] and z.tt_norm() == 0.0
    t = tt.TensorTrain(P.random_tt([3] * 4, 3, seed=1))
    with pytest.raises(ValueError):
        t.truncate(max_rank=0)
    with pytest.raises(ValueError):
        t.truncate(max_rank=-2)

"""Rounded cores own the storage of their entries and no more; a train of one core
does not go to the batched kernel."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def test_one_core_is_left_to_the_sweeps():
    from ttnumpy_b200 import tensor_train as T

    assert T.round_in_one_launch([torch.ones(1, 8, 1, 1, dtype=torch.float64)], 1e-8, None) is None


@pytest.mark.gpu
def test_one_core_train_is_refused_by_truncate():
    """As the truncation of the host divides the error among no bonds."""
    import ttnumpy_b200 as tt

    x = tt.tt_svd(np.arange(8.0), 1e-12, physical_indexes=[8])
    assert len(x) == 1
    x.orth_center = None
    with pytest.raises(ZeroDivisionError):
        x.truncate(1e-8)


@pytest.mark.gpu
@pytest.mark.parametrize("n,r", [(64, 12), (3, 4)])
@pytest.mark.parametrize("canonical", ["auto", "left", "right"])
def test_cores_own_their_entries(n, r, canonical):
    import ttnumpy_b200 as tt
    from ttnumpy_b200 import problems

    x = tt.TensorTrain(problems.random_tt([n] * 4, r, seed=1))
    y = (x + x).truncate(1e-10, canonical=canonical)
    assert y.max_rank <= r
    for c in y.cores:
        assert c.is_contiguous()
        assert c.untyped_storage().nbytes() == 8 * c.numel()
    z = (x + x).orthonormalize().compress_svd(1e-10)
    for c in z.cores:
        assert c.untyped_storage().nbytes() == 8 * c.numel()

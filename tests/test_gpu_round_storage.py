"""Rounded cores own the storage of their entries and no more."""

import pytest

pytest.importorskip("torch")


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

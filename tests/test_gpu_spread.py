"""A batch that leaves the device idle is spread over clusters of blocks with
the lone blocks' bits."""

import numpy as np
import pytest

from ttnumpy_b200 import persistent as P


@pytest.mark.parametrize("count,size", [(1, 8), (8, 8), (9, 8), (10, 4), (18, 4), (19, 2), (37, 2),
                                        (38, 1), (256, 1)])
def test_spread_keeps_half_of_the_device(count, size):
    assert P.spread(count, 148) == size


@pytest.mark.gpu
@pytest.mark.parametrize("mode,direct", [(21, 150), (21, 511), (21, 1024), (32, 1000)])
def test_spread_equals_lone_blocks(mode, direct):
    """Products, vector passes, eliminations (also of the smallest and largest
    systems that are shared) and the residual norm's tall factorisations give
    the same bits on a cluster."""
    from ttnumpy_b200 import problems

    kw = dict(residual_tol=1e-8, symmetric=True, max_sweeps=5, seed=0, stagnation_factor=None,
              direct_solve_size=direct, kickrank=3)
    theta = np.array([0.3, -0.7, 0.5, 0.9])
    probs = [problems.parametric_diffusion(4, mode, theta), problems.qtt_poisson_2d(7)]
    reqs = [(p.A, p.b, None, kw) for p in probs]
    lone = P.PersistentBatch(P.prepare(reqs), 64, cluster=1).run()
    for a, b in zip(lone, P.amen_persistent(reqs)):
        assert a.status == 0 and b.status == 0
        assert a.info.residuals == b.info.residuals
        assert all(np.array_equal(u, v) for u, v in zip(a.x.to_numpy(), b.x.to_numpy()))

"""Whole solves whose cores have as many rows as a warp-per-column Householder
step takes at most (33, 65, 129: one, two, four rows of a lane), and one more."""

import numpy as np
import pytest

from oracle import tt_oracle as O
from ttnumpy_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r", [(11, 3), (17, 2), (13, 5), (11, 6), (43, 3), (10, 13)])
def test_solve_with_cores_of_n_times_r_rows(n, r):
    from ttnumpy_b200 import persistent

    p = problems.parametric_diffusion(3, n, np.array([0.4, -0.6, 0.8]))
    x0 = problems.random_tt([n] * 3, r, 5)
    kw = dict(residual_tol=1e-8, symmetric=True, max_sweeps=15, seed=0, stagnation_factor=None)
    (res,) = persistent.amen_persistent([(p.A, p.b, x0, kw)])
    assert res.status == 0 and res.info.converged
    x = O.Train(res.x.to_numpy(), res.x.orth_center)
    assert O.relative_residual(O.Train(p.A), O.Train(p.b), x) <= 1.05e-8

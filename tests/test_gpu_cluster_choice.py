"""Thread blocks per solve of ``amen_persistent``: the number asked for, one
block being one, and a spread batch only where none is asked for."""

import types

import numpy as np
import pytest

from ttnumpy_b200 import persistent as P


@pytest.mark.parametrize("cluster,sizes", [(None, [4, 8]), (1, [1, 1]), (2, [2, 2]), (8, [8, 8])])
def test_blocks_per_solve(monkeypatch, cluster, sizes):
    """Ten requests on 148 multiprocessors, nine solved in the first launch."""
    seen = []

    class Batch:
        def __init__(self, preps, rmax, time_limit=None, cluster=1):
            seen.append(cluster)
            self.preps, self.rmax = preps, rmax

        def run(self, stream=None):
            return [types.SimpleNamespace(status=-4 if p == 7 and self.rmax == 64 else 0)
                    for p in self.preps]

    monkeypatch.setattr(P, "PersistentBatch", Batch)
    monkeypatch.setattr(P, "prepare", list)
    monkeypatch.setattr(P.K, "device_ok", lambda: None)
    monkeypatch.setattr(P.torch.cuda, "get_device_properties",
                        lambda *_: types.SimpleNamespace(multi_processor_count=148))
    kw = {} if cluster is None else {"cluster": cluster}
    out = P.amen_persistent(list(range(10)), **kw)
    assert [r.status for r in out] == [0] * 10
    assert seen == sizes


@pytest.mark.gpu
def test_lone_block_equals_clusters():
    """A mode-64 diffusion solve, a mode-32 one and a QTT one: one block each,
    spread, and on clusters of four, the same bits."""
    from ttnumpy_b200 import problems

    kw = dict(residual_tol=1e-8, symmetric=True, max_sweeps=6, seed=0, stagnation_factor=None)
    probs = [problems.parametric_diffusion(4, 64, np.array([0.2, -0.5, 0.8, 0.1])),
             problems.parametric_diffusion(5, 32, np.array([0.2, -0.5, 0.8, 0.1, -0.9])),
             problems.qtt_poisson_2d(6)]
    reqs = [(p.A, p.b, None, kw) for p in probs]
    lone = P.amen_persistent(reqs, rmax=96, cluster=1)
    for other in (P.amen_persistent(reqs, rmax=96), P.amen_persistent(reqs, rmax=96, cluster=4)):
        for a, b in zip(lone, other):
            assert a.status == 0 and b.status == 0
            assert a.info.residuals == b.info.residuals
            assert all(np.array_equal(u, v) for u, v in zip(a.x.to_numpy(), b.x.to_numpy()))

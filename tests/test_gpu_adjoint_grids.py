"""One adjoint initialised again and again: across grids whose rebuilds count and
grids of so many cells that they sort by digits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rollout(a, scene, size):
    pos, vel, _, _, prm, _ = scene
    gx = np.zeros_like(pos)
    gx[:, :3] = np.random.default_rng(4).standard_normal((len(pos), 3)) / len(pos)
    a.initialize(len(pos), (0.0, 0.0, 0.0), size, prm, max_neighbors=128, checkpoint_every=2)
    a.forward(pos, vel, 3)
    return a.backward(gx, np.zeros_like(gx))


def test_again_on_other_grids(pbf, scenes):
    a = pbf.PBFAdjoint()
    for n, size in ((9, (2.0, 1.0, 1.0)), (6, (12.0, 9.0, 9.0)), (7, (12.0, 9.0, 9.0)),
                    (11, (2.0, 1.0, 1.0)), (9, (4.0, 4.0, 4.0))):
        scene = scenes.dam_break(n, n, n, (12.0, 9.0, 9.0), seed=n)
        got = _rollout(a, scene, size)
        fresh = pbf.PBFAdjoint()
        for g, w in zip(got, _rollout(fresh, scene, size)):
            np.testing.assert_array_equal(g, w)
        fresh.close()
    a.close()


def test_initialize_that_runs_out_of_memory(pbf, scenes):
    """The adjoint is as if never initialised, until an initialise succeeds."""
    scene = scenes.dam_break(9, 9, 9, (2.0, 1.0, 1.0), seed=1)
    pos, vel, _, _, prm, _ = scene
    a = pbf.PBFAdjoint()
    want = _rollout(a, scene, (2.0, 1.0, 1.0))
    with pytest.raises(pbf.SolverRuntimeError, match="out of memory"):
        a.initialize(len(pos), (0.0, 0.0, 0.0), (2.0, 1.0, 1.0), prm, max_neighbors=1 << 28)
    with pytest.raises(pbf.LogicError):
        a.forward(pos, vel, 1)
    with pytest.raises(pbf.LogicError):
        a.backward(pos, vel)
    for g, w in zip(_rollout(a, scene, (2.0, 1.0, 1.0)), want):
        np.testing.assert_array_equal(g, w)
    a.close()

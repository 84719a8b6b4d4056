"""The adjoint's gather passes at list lengths of no, one and a few entries a
lane and where their lanes per particle change, and its graphs across changes of the physics.

Each gradient is checked along a random direction in v0 against the FP64
forward-mode tangents of the same step, to 1e-3 as elsewhere.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(scenes, n):
    side = max(2, int(np.ceil(n ** (1.0 / 3.0))))
    box = (2 * side * 0.05, 1.5 * side * 0.05, 2 * side * 0.05)
    pos, _, mn, mx, prm, _ = scenes.dam_break(side, side, side, box, seed=n)
    pos = pos[:n]
    vel = np.zeros_like(pos)
    vel[:, 0] = 0.4 * np.sin(3.0 * pos[:, 1])
    vel[:, 1] = 0.4 * np.cos(2.0 * pos[:, 2])
    vel[:, 2] = 0.4 * np.sin(2.5 * pos[:, 0])
    return pos, vel, mn, mx, prm


def _gradient(pbf, scene, gx, rest_density=None):
    pos, vel, mn, mx, prm = scene
    a = pbf.PBFAdjoint()
    a.initialize(len(pos), mn, mx, prm, max_neighbors=128, checkpoint_every=1)
    if rest_density is not None:
        a.set_physics(rest_density, prm.xsphViscosity)
    a.forward(pos, vel, 1)
    out = a.backward(gx, np.zeros_like(gx))
    a.close()
    return out


def _gx(n):
    g = np.zeros((n, 4), np.float32)
    g[:, :3] = np.random.default_rng(n + 1).standard_normal((n, 3)) / n
    return g


@pytest.mark.parametrize("n", [1, 2, 33, 4097, 131071, 131072])
def test_gradient_at_lane_boundaries(pbf, scenes, orc, n):
    scene = _scene(scenes, n)
    pos, vel, mn, mx, prm = scene
    gx = _gx(n)
    _, gv0, _, _ = _gradient(pbf, scene, gx)
    r = np.random.default_rng(n + 2).standard_normal((1, n, 3))
    # Directions with a component along the gradient, so that the derivative
    # is no small difference of large terms.
    r[0] += gv0[:, :3] * (np.sqrt(n) / np.linalg.norm(gv0[:, :3]))
    _, _, tx, _ = orc.diff_rollout(pos, vel, prm.as_dict(), mn, mx, 1, tv0=r)
    want = float((gx[:, :3].astype(np.float64) * tx[0]).sum())
    got = float((gv0[:, :3].astype(np.float64) * r[0]).sum())
    assert abs(got - want) <= 1e-3 * abs(want)


def test_physics_changes_reach_the_graphs(pbf, scenes):
    scene = _scene(scenes, 700)
    pos, vel, mn, mx, prm = scene
    gx = _gx(700)
    a = pbf.PBFAdjoint()
    a.initialize(700, mn, mx, prm, max_neighbors=128, checkpoint_every=1)
    rho = prm.restDensity
    for density in (rho, rho, 0.97 * rho, rho, 1.02 * rho):
        a.set_physics(density, prm.xsphViscosity)
        with pytest.raises(pbf.LogicError):
            a.backward(gx, np.zeros_like(gx))  # the recorded forward is dropped
        a.forward(pos, vel, 1)
        got = a.backward(gx, np.zeros_like(gx))
        for g, w in zip(got, _gradient(pbf, scene, gx, density)):
            np.testing.assert_array_equal(g, w)
    a.close()

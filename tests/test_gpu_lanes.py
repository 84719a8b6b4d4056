"""The lane-group kernels at the sizes and lengths where they change.

Groups of 32, 16 and 8 lanes by default up to 3,072, 10,240 and 18,432
particles, one thread per particle above, and 2, 4 or 8 when set; walks of
nine lanes with three particles a warp.  A packed core (rows of more than 32
and more than 64 candidates, lists longer than a 64-entry stash) inside a
loose block: two frames equal the FP32 oracle bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(n, 0) for n in (1, 2, 3, 4, 31, 97, 3072, 3073, 10240, 10241, 18432, 18433, 22528,
                         22529)]
SIZES += [(n, lanes) for lanes in (2, 4, 8) for n in (1, 5, 1000)]


def _scene(n, rng):
    core = min(n // 2, 400)
    side = max(1, round((n - core) ** (1.0 / 3.0)))
    at = np.arange(n - core)
    pos = np.ones((n, 4), np.float32)
    loose = np.stack([at % side, at // side % side, at // (side * side)], 1) * 0.06
    pos[:n - core, :3] = 0.05 + loose + rng.uniform(-0.01, 0.01, loose.shape)
    k = np.arange(core)
    packed = np.stack([k % 8, k // 8 % 8, k // 64], 1) * 0.027
    pos[n - core:, :3] = 0.06 + packed + rng.uniform(-0.004, 0.004, packed.shape)
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0.0, 0.3, (n, 3))
    hi = tuple(float(v) for v in pos[:, :3].max(0) + 0.25)
    order = rng.permutation(n)
    return pos[order], vel[order], hi


@pytest.mark.parametrize("n,lanes", SIZES)
def test_lane_groups_match_oracle(pbf, scenes, orc, n, lanes):
    pos, vel, hi = _scene(n, np.random.default_rng(n + 1000 * lanes))
    prm = scenes.dam_break_params()
    prm.lambdaEpsilon = 1e6
    prm.solverIterations = 2
    s = pbf.PBFSolver()
    s.initialize(n, (0.0, 0.0, 0.0), hi, prm)
    s.set_walk_lanes(lanes)
    s.set_particles(pos, vel)
    s.run(2)
    o = orc.OracleSolver(32)
    o.initialize(n, (0.0, 0.0, 0.0), hi, prm.as_dict())
    o.set_particles(pos, vel)
    assert o.run(2) == 0
    _, wid, wcnt = s.working_state()
    _, oid, ocnt = o.working()
    np.testing.assert_array_equal(wid, oid)
    np.testing.assert_array_equal(wcnt, ocnt)
    for got, want in ((s.copy_positions_to_host(), o.positions()),
                      (s.copy_velocities_to_host(), o.velocities())):
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    s.close()

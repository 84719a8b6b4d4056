"""The one-thread-per-particle walks at the lengths of their queues.

A lane queues up to 12 chunks of 32 candidates with hits, and a warp empties
its queues when any is full.  Blocks of particles at spacings with 30 to 250
neighbours (from fewer than 12 such chunks to several times as many), alone
or beside loose ones in the same warp, with warps that are not full, lists
slot-major and compact: two frames equal the FP32 oracle bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("spacing", [0.05, 0.036, 0.03, 0.0265])
@pytest.mark.parametrize("n", [1, 31, 33, 96, 700, 2049])
def test_walks_match_oracle(pbf, scenes, orc, n, spacing, compact):
    rng = np.random.default_rng(n + round(spacing * 1e5))
    k = np.arange(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = np.stack([k % 10, k // 10 % 10, k // 100], 1) * spacing + 0.07
    pos[:, :3] += rng.uniform(-0.1, 0.1, (n, 3)) * spacing
    loose = n // 3
    pos[:loose, :3] += rng.uniform(0.0, 0.5, (loose, 3))
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0.0, 0.3, (n, 3))
    hi = tuple(float(v) for v in pos[:, :3].max(0) + 0.25)
    prm = scenes.dam_break_params()
    prm.lambdaEpsilon = 1e6
    prm.solverIterations = 2
    s = pbf.PBFSolver()
    s.initialize(n, (0.0, 0.0, 0.0), hi, prm, list_capacity=n * 300 if compact else None)
    s.set_walk_lanes(1)
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

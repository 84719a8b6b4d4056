"""The step's counting sort by cell at the grid sizes where it changes.

Up to 8,192 cells one launch scans the counts in every block; up to 32,768 a
scan's blocks sum the counts before them; above, tile sums come from a launch
of their own, with larger tiles above 2^20; with far more cells than particles
the radix sort orders them.
Shuffled particles, some alone, some dozens to a cell, some outside the
grid: after two frames the working order (stable within a cell), the counts
and the state equal the FP32 oracle's bit for bit, also on a solver whose last
run failed half way.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# dims, particles: 1 cell; 8,191 to 8,193 cells; 32,768 and 32,769; whole
# tiles; more than 2^20 cells; more than 8 n + 65,536 cells.
GRIDS = [((1, 1, 1), 1), ((1, 1, 1), 190), ((8191, 1, 1), 1025), ((32, 16, 16), 1024),
         ((2731, 3, 1), 2047), ((32, 32, 32), 3000), ((331, 11, 9), 1500), ((64, 36, 32), 5000),
         ((73, 70, 3), 300), ((128, 128, 65), 125000), ((100, 100, 10), 700)]


def _scene(dims, n):
    rng = np.random.default_rng(n * 31 + dims[0])
    hi = np.asarray(dims) * 0.1 * 0.9999
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform((0.0, 0.0, 0.0), hi, (n, 3))
    clump = rng.uniform((0.0, 0.0, 0.0), hi, (max(8, n // 128), 3))
    k = n // 2
    pos[:k, :3] = clump[rng.integers(0, len(clump), k)] + rng.uniform(-0.02, 0.02, (k, 3))
    pos[k:k + n // 16, 1] += np.float32(hi[1] + 0.3)  # above the open top
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0.0, 1.0, (n, 3))
    order = rng.permutation(n)
    return pos[order], vel[order], tuple(float(v) for v in hi)


@pytest.mark.parametrize("dims,n", GRIDS)
def test_reorder_matches_oracle(pbf, scenes, orc, dims, n):
    pos, vel, hi = _scene(dims, n)
    assert pbf.grid_dims((0, 0, 0), hi, 0.1) == dims
    prm = scenes.dam_break_params()
    prm.lambdaEpsilon = 1e6
    s = pbf.PBFSolver()
    s.initialize(max(n, 300), (0.0, 0.0, 0.0), hi, prm)
    # A run that fails in its first walk (300 particles in one place).
    s.set_particles(np.full((300, 4), 0.05, np.float32), np.zeros((300, 4), np.float32))
    with pytest.raises(pbf.NeighborOverflowError):
        s.run(1)
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

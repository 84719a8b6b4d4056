"""Compact lists in slices of 32 particles and, where those would not fit,
back to back: the smallest capacity that holds the lists still steps, one
entry less overflows, and every layout gives the slot-major result."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 2047, 2049, 5000])
def test_layouts_agree_down_to_the_smallest_capacity(pbf, scenes, n):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    at = np.arange(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = 0.03 + 0.05 * np.stack([at % side, at // side % side, at // side ** 2], 1)
    pos[:, :3] += rng.uniform(-0.01, 0.01, (n, 3))
    pos[: n // 8, :3] = pos[0, :3] + rng.uniform(-0.04, 0.04, (n // 8, 3)) * (n / 5000.0)
    vel = np.zeros_like(pos)
    hi = tuple(float(v) for v in pos[:, :3].max(0) + 0.3)
    prm = scenes.dam_break_params()
    prm.lambdaEpsilon = 1e6

    def run(cap):
        s = pbf.PBFSolver()
        s.initialize(n, (0.0, 0.0, 0.0), hi, prm, max_neighbors=1024, list_capacity=cap)
        s.set_particles(pos, vel)
        try:
            s.run(1)
            return s.copy_positions_to_host(), s.copy_velocities_to_host()
        except pbf.NeighborOverflowError:
            return None
        finally:
            s.close()

    want = run(None)
    low, high = 0, n * 1024  # overflows / fits
    while high - low > 1:
        mid = (low + high) // 2
        if run(mid) is None:
            low = mid
        else:
            high = mid
    for cap in (high, high + high // 50, 2 * high, n * 1024):
        for got, ref in zip(run(cap), want):
            np.testing.assert_array_equal(got.view(np.uint32), ref.view(np.uint32))

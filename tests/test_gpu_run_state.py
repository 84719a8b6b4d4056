"""The state that a run expects cleared (status, the counting sort's counts, the
compact lists' control words) when nothing has run on it yet: status checks on a
fresh or re-initialised solver, in every form, leave the first run's result the
FP32 oracle's bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHECKS = {
    "synchronize": lambda s: s.synchronize(),
    "time_no_frames": lambda s: s.time_frames(0),
    "run_no_frames": lambda s: (s.run_async(0), s.synchronize()),
}


def _scene(side, height, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(side * height * side)
    pos = np.ones((len(k), 4), np.float32)
    pos[:, :3] = np.stack([k % side, k // side % height, k // (side * height)], 1) * 0.05 + 0.03
    pos[:, :3] += rng.uniform(-0.004, 0.004, (len(k), 3))
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0.0, 0.2, (len(k), 3))
    return pos, vel, (2.0 * side * 0.05, height * 0.06, side * 0.05 + 0.06)


def _oracle(orc, prm, pos, vel, hi, frames):
    o = orc.OracleSolver(32)
    o.initialize(len(pos), (0.0, 0.0, 0.0), hi, prm.as_dict())
    o.set_particles(pos, vel)
    assert o.run(frames) == 0
    return o


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("check", list(CHECKS))
@pytest.mark.parametrize("where", ["before", "after"])
def test_status_check_before_the_first_run(pbf, scenes, orc, compact, check, where):
    prm = scenes.dam_break_params()
    s = pbf.PBFSolver()
    # A grid of more cells first, so that the second one's buffers are used memory.
    for side, height, seed in ((20, 24, 1), (12, 10, 2)):
        pos, vel, hi = _scene(side, height, seed)
        s.initialize(len(pos), (0.0, 0.0, 0.0), hi, prm,
                     list_capacity=64 * len(pos) if compact else None)
        if where == "before":
            CHECKS[check](s)
        s.set_particles(pos, vel)
        if where == "after":
            CHECKS[check](s)
        s.run(2)
        o = _oracle(orc, prm, pos, vel, hi, 2)
        for got, want in ((s.copy_positions_to_host(), o.positions()),
                          (s.copy_velocities_to_host(), o.velocities())):
            np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    s.close()

"""What can be asked of a solver whose last run failed."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clump(n):
    """n particles in one place: more neighbours than any list holds."""
    return np.full((n, 4), 0.05, np.float32), np.zeros((n, 4), np.float32)


def test_copies_stay_inside_their_destination(pbf, scenes):
    torch = pytest.importorskip("torch")
    pos, vel, mn, mx, prm, _ = scenes.dam_break_16k()
    s = pbf.PBFSolver()
    s.initialize(4096, mn, mx, prm)
    s.set_particles(pos[:4096], vel[:4096])
    s.run(2)  # both id buffers in use
    s.set_particles(*_clump(300))
    with pytest.raises(pbf.NeighborOverflowError):
        s.run(1)
    out = torch.full((4096, 4), -7.0, device="cuda")
    torch.cuda.synchronize()
    s.copy_positions_device(out[:300])
    s.copy_velocities_device(out[:300])
    assert bool((out[300:] == -7.0).all())
    s.set_particles(pos[:300], vel[:300])
    s.copy_positions_device(out[:300])
    np.testing.assert_array_equal(out[:300].cpu().numpy(), pos[:300])
    s.close()

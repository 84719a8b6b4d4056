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


@pytest.mark.parametrize("entries", [1, 2, 4, 20])
def test_density_of_lists_without_a_place(pbf, scenes, entries):
    """Compact lists of too small a capacity: the density error of what the failed
    run left (any number) can be asked for, and the next run is right."""
    pos, vel, mn, mx, prm, _ = scenes.dam_break_16k()
    n = len(pos)
    s = pbf.PBFSolver()
    s.initialize(n, mn, mx, prm, list_capacity=entries * n)  # some 30 needed
    for _ in range(2):
        s.set_particles(pos, vel)
        with pytest.raises(pbf.NeighborOverflowError, match="compact list capacity"):
            s.run(1)
        assert len(s.density_error()) == 2
    few = 1000
    s.set_particles(pos[::16][:few], vel[:few])
    s.run(2)
    f = pbf.PBFSolver()
    f.initialize(n, mn, mx, prm)
    f.set_particles(pos[::16][:few], vel[:few])
    f.run(2)
    assert s.density_error() == f.density_error()
    np.testing.assert_array_equal(s.copy_positions_to_host(), f.copy_positions_to_host())
    s.close()
    f.close()

"""Device arrays handed to the solver: taken by a kernel where they are
16-byte aligned memory of its device, copied otherwise, with the same result;
a rejected array leaves the particles as they were."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 3000])
@pytest.mark.parametrize("offset", [0, 4, 1, 3])
def test_device_arrays_aligned_or_not(pbf, scenes, n, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.05, 1.5, (n, 3))
    vel = rng.normal(0.0, 0.1, (n, 4)).astype(np.float32)
    s = pbf.PBFSolver()
    s.initialize(n, (0.0, 0.0, 0.0), (1.6, 1.6, 1.6), scenes.dam_break_params())

    def array():
        return torch.zeros(4 * n + 8, device="cuda")[offset:offset + 4 * n].view(n, 4)

    p, v, po, vo = array(), array(), array(), array()
    p.copy_(torch.from_numpy(pos))
    v.copy_(torch.from_numpy(vel))
    torch.cuda.synchronize()
    s.set_particles_device(p, v)
    s.copy_positions_device(po)
    s.copy_velocities_device(vo)
    np.testing.assert_array_equal(po.cpu().numpy(), pos)
    np.testing.assert_array_equal(vo.cpu().numpy(), vel)
    bad = p.clone()
    bad[n // 2, 1] = float("nan")
    torch.cuda.synchronize()
    with pytest.raises(pbf.InvalidArgument):
        s.set_particles_device(bad, v)
    np.testing.assert_array_equal(s.copy_positions_to_host(), pos)
    np.testing.assert_array_equal(s.copy_velocities_to_host(), vel)
    s.close()

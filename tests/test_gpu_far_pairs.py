"""Listed pairs whose difference overflows to infinity.  The kernels' gradients are
zero outside the radius, so such a pair adds nothing: the stage calls that take
the caller's lists equal the FP32 oracle bit for bit."""

import numpy as np
import pytest

from backends import CudaBackend, OracleBackend

pytestmark = pytest.mark.gpu

H = 0.5


def _setup(far, entries):
    """Particle 0 with the listed entries; the others have no lists."""
    pos = np.ones((5, 4), np.float32)
    pos[:, :3] = [[1.0, 1.0, 1.0], [1.1, 1.2, 0.9], [0.8, 1.0, 1.1], [1.0, 1.0, 1.0],
                  [1.0, 1.0, 1.0]]
    pos[3, :3] = far
    pos[0, :3] += np.asarray([-3e38 if abs(v) > 1e38 else 0.0 for v in far], np.float32)
    rng = np.random.default_rng(3)
    vel = rng.normal(0.0, 1.0, (5, 4)).astype(np.float32)
    nb = np.zeros((4, 5), np.uint32)
    nb[:len(entries), 0] = entries
    cnt = np.asarray([len(entries), 0, 0, 0, 0], np.int32)
    return pos, vel, nb.ravel(), cnt


FAR = [(3e38, 1.0, 1.0), (1.0, 3e38, 3e38), (3e38, 3e38, 3e38), (1e30, -1e30, 1.0),
       (1.0, 1.0, 1.0)]


@pytest.mark.parametrize("far", FAR)
@pytest.mark.parametrize("entries", [(3,), (1, 3), (3, 3, 2), (1, 2, 3, 4)])
def test_lambda(orc, far, entries):
    pos, _, nb, cnt = _setup(far, entries)
    got, want = (B.lam(pos, nb, cnt, 4, 5, H, 1.0, 1000.0, 100.0)
                 for B in (CudaBackend(), OracleBackend()))
    assert np.isfinite(want).all()
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("far", FAR)
def test_one_neighbour(orc, far):
    pos, vel, nb, cnt = _setup(far, (3,))
    lam = np.asarray([-0.1, 0.2, 0.3, 0.4, 0.5], np.float32)
    om = np.abs(vel[::-1])
    for stage in (lambda B: B.delta(pos, nb, cnt, 4, lam, 5, H, 1.0, 1000.0, 0.001, 4, 0.1),
                  lambda B: B.vorticity(pos, vel, nb, cnt, 4, 5, H),
                  lambda B: B.confinement(pos, nb, cnt, 4, om, vel, 5, H, 0.01, 0.1)):
        got, want = stage(CudaBackend()), stage(OracleBackend())
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(np.asarray(got).view(np.uint32),
                                      np.asarray(want).view(np.uint32))

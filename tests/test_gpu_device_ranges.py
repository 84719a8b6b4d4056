"""Device arrays that are shorter than the particle count: refused with a status
on the host, with the solver's particles (and a destination) as they were, and
taken where they fit their allocation exactly or lie inside it."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 262_144
BYTES = 16 * N


class Driver:
    """Raw device allocations, so that the end of an array is the end of its
    allocation."""

    def __init__(self):
        self.lib = C.CDLL("libcuda.so.1")
        self.held = []

    def range(self, ptr):
        base, size = C.c_uint64(), C.c_size_t()
        st = self.lib.cuMemGetAddressRange_v2(C.byref(base), C.byref(size), C.c_uint64(ptr))
        return (base.value, size.value) if st == 0 else None

    def alloc(self, nbytes):
        """An allocation with nothing behind it."""
        for _ in range(32):
            p = C.c_uint64()
            assert self.lib.cuMemAlloc_v2(C.byref(p), C.c_size_t(nbytes)) == 0
            self.held.append(p.value)
            if self.range(p.value) == (p.value, nbytes) and self.range(p.value + nbytes) is None:
                return p.value
        pytest.skip("device allocations stand side by side")

    def put(self, ptr, a):
        a = np.ascontiguousarray(a)
        assert self.lib.cuMemcpyHtoD_v2(C.c_uint64(ptr), a.ctypes.data_as(C.c_void_p),
                                        C.c_size_t(a.nbytes)) == 0

    def get(self, ptr, n):
        a = np.empty((n, 4), np.float32)
        assert self.lib.cuMemcpyDtoH_v2(a.ctypes.data_as(C.c_void_p), C.c_uint64(ptr),
                                        C.c_size_t(a.nbytes)) == 0
        return a

    def close(self):
        for p in self.held:
            self.lib.cuMemFree_v2(C.c_uint64(p))


class Array:
    def __init__(self, ptr):
        self.ptr, self.shape = ptr, (N, 4)

    def data_ptr(self):
        return self.ptr


@pytest.fixture
def setup(pbf, scenes):
    rng = np.random.default_rng(9)
    pos = np.ones((N, 4), np.float32)
    pos[:, :3] = rng.uniform(0.05, 3.0, (N, 3))
    vel = rng.normal(0.0, 0.1, (N, 4)).astype(np.float32)
    s = pbf.PBFSolver()
    s.initialize(N, (0.0, 0.0, 0.0), (3.2, 3.2, 3.2), scenes.dam_break_params(), 1)
    s.set_particles(pos, vel)
    d = Driver()
    yield s, d, pos, vel
    s.close()
    d.close()


@pytest.mark.parametrize("offset", [0, 4096])
def test_arrays_that_fit(setup, offset):
    s, d, pos, vel = setup
    p, v, out = (d.alloc(BYTES + offset) + offset for _ in range(3))
    d.put(p, vel)
    d.put(v, pos)
    s.set_particles_device(Array(p), Array(v))
    s.copy_velocities_device(Array(out))
    np.testing.assert_array_equal(d.get(out, N), pos)
    s.copy_positions_device(Array(out))
    np.testing.assert_array_equal(d.get(out, N), vel)


@pytest.mark.parametrize("nbytes", [BYTES // 2, 4096])
@pytest.mark.parametrize("which", ["positions", "velocities", "destination"])
def test_short_arrays_are_refused(pbf, setup, which, nbytes):
    s, d, pos, vel = setup
    whole = d.alloc(BYTES)
    short = d.alloc(nbytes)  # last: nothing comes to stand behind it
    d.put(short, vel[:nbytes // 16])
    d.put(whole, vel)
    with pytest.raises(pbf.SolverRuntimeError, match="invalid argument"):
        if which == "positions":
            s.set_particles_device(Array(short), Array(whole))
        elif which == "velocities":
            s.set_particles_device(Array(whole), Array(short))
        else:
            s.copy_positions_device(Array(short))
    np.testing.assert_array_equal(s.copy_positions_to_host(), pos)
    np.testing.assert_array_equal(s.copy_velocities_to_host(), vel)
    np.testing.assert_array_equal(d.get(short, nbytes // 16), vel[:nbytes // 16])

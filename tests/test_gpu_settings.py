"""Settings that change no result: which kernels they run, by name."""

import pytest

pytestmark = pytest.mark.gpu


def _solver(pbf, scenes, n):
    pos, vel, mn, mx, prm, _ = scenes.dam_break_16k()
    s = pbf.PBFSolver()
    s.initialize(n, mn, mx, prm)
    s.set_particles(pos[:n], vel[:n])
    s.step()
    return s


def _launched(call):
    """Names of the kernels that call() launches, each as often as it ran."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    for _ in range(2):  # a process's first trace may come back empty
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            call()
        names = [e.name.split("(float")[0] for e in p.events() if "pbf::" in e.name]
    assert names
    return sorted(names)


@pytest.mark.parametrize("n", [1000, 3072, 3073, 10240, 10241, 16384])
def test_setting_the_lanes_read_changes_no_kernel(pbf, scenes, n):
    s = _solver(pbf, scenes, n)
    default = _launched(s.step)
    assert any("_group<" in k for k in default)
    s.set_walk_lanes(s.walk_lanes())
    assert _launched(s.step) == default
    s.close()

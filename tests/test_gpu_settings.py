"""Settings that change no result: which kernels they run, by name."""

import pytest

pytestmark = pytest.mark.gpu


def _solver(pbf, scenes, n, size=None):
    pos, vel, mn, mx, prm, _ = scenes.dam_break_16k()
    mx = mx if size is None else (size, size, size)
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


@pytest.mark.parametrize("size,tiles", [(2.0, 0), (10.0, 2)])
def test_autotune_tries_what_the_frames_run(pbf, scenes, size, tiles):
    """Six kernels at four block sizes, and the sort's tiles only in a grid of so
    many cells that the rebuilds sort by digits; two untimed frames and one."""
    s = _solver(pbf, scenes, 1000, size)
    frames = _launched(lambda: s.autotune(1))
    assert any("k_bin_gather" in k for k in frames) == (tiles == 0)
    assert sum("k_predict" in k for k in frames) == (6 * 4 + tiles) * 3
    assert s.block_sizes()["sort_tile"] in ((1024,) if tiles == 0 else (1024, 4096))
    s.close()

"""The allocation-free grid build by counting, at the sizes where it changes.

One cell; whole and ragged tiles of the count scan; more than 2^20 cells; cells
of 256 positions (ranked by themselves) and 257 (by their bits), 8,193 (in two
parts), 65,536 and 65,537 (from the list, from the keys); the last cell counts
that are counted, with the cells and with the positions, and one beyond (radix
sort); the cell arrays 4-byte aligned only.  All outputs equal the oracle's.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# dims, positions, positions per clump (0: none)
BUILDS = [((1, 1, 1), 1, 0), ((1, 1, 1), 262144, 0), ((1023, 1, 1), 5000, 256),
          ((32, 32, 1), 5140, 257), ((41, 25, 1), 3000, 100), ((64, 60, 48), 200003, 1000),
          ((128, 128, 64), 131072, 0), ((1048577, 1, 1), 131072, 300), ((67, 1000, 1), 183, 0),
          ((67001, 1, 1), 183, 100), ((16, 16, 16), 262144, 0), ((16, 16, 15), 262144, 0),
          ((64, 60, 48), 262144, 131072), ((64, 60, 48), 200003, 65537),
          ((64, 60, 48), 262143, 65536), ((64, 60, 48), 70001, 8193)]


@pytest.mark.parametrize("dims,n,clump", BUILDS)
def test_counting_build_matches_oracle(pbf, orc, dims, n, clump):
    torch = pytest.importorskip("torch")
    L = pbf.load()
    rng = np.random.default_rng(n + dims[0])
    lo, cell = (0.0, 0.0, 0.0), 1.0
    hi = tuple(float(d) for d in dims)
    assert pbf.grid_dims(lo, hi, cell) == dims
    pos = np.ones((n, 4), np.float32)
    # Some outside the grid, which its border cells take.
    pos[:, :3] = rng.uniform(-0.5, np.asarray(hi) + 0.5, (n, 3))
    if clump:
        k = n // 2 // clump * clump
        at = rng.choice(np.prod(dims), k // clump, replace=False)
        at = np.stack([at % dims[0], at // dims[0] % dims[1], at // (dims[0] * dims[1])], 1)
        pos[:k, :3] = np.repeat(at, clump, 0) + rng.uniform(0.1, 0.9, (k, 3))
        pos = pos[rng.permutation(n)]
    want = orc.grid_build(pos, lo, cell, dims)
    cells = int(np.prod(dims))
    d_pos = torch.from_numpy(pos).cuda()
    d_sk, d_si = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    d_cs, d_ce = (torch.full((cells + 2,), 123, dtype=torch.int32, device="cuda")
                  for _ in range(2))
    torch.cuda.synchronize()
    for _ in range(2):
        assert L.pbf_grid_build_static_scratch(
            C.c_void_p(d_pos.data_ptr()), n, pbf.Float3(*lo), pbf.Float3(*hi), cell,
            C.c_void_p(d_sk.data_ptr()), C.c_void_p(d_si.data_ptr()),
            C.c_void_p(d_cs[1:].data_ptr()), C.c_void_p(d_ce[1:].data_ptr()), None) == 0
        torch.cuda.synchronize()
        got = (d_sk.cpu().numpy().view(np.uint32), d_si.cpu().numpy().view(np.uint32),
               d_cs.cpu().numpy()[1:-1], d_ce.cpu().numpy()[1:-1])
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    assert d_cs[0] == 123 and d_cs[-1] == 123 and d_ce[0] == 123 and d_ce[-1] == 123

"""The neighbour walk where the search radius reaches past thin grids.

Lists equal the FP32 oracle's slot for slot, and a walk takes no longer than its
grid has rows: in a grid one cell wide and deep the call costs the same whether
the radius is one cell or all of them.
"""

import time

import numpy as np
import pytest

from backends import CudaBackend, OracleBackend

pytestmark = pytest.mark.gpu


def _search(B, pos, dims, cell, h, max_nb=256):
    hi = tuple((d - 0.5) * cell for d in dims)
    assert tuple(B.grid_dims((0.0, 0.0, 0.0), hi, cell)) == dims
    _, perm, cs, ce = B.grid_build(pos, (0.0, 0.0, 0.0), hi, cell)
    return B.find_neighbors(pos[perm], cs, ce, dims, (0.0, 0.0, 0.0), cell, h, max_nb)


@pytest.mark.parametrize("dims", [(40, 1, 1), (1, 40, 1), (1, 1, 40), (5, 40, 1), (64, 2, 1),
                                  (2, 1, 33), (7, 6, 5)])
@pytest.mark.parametrize("radius", [1, 2, 8, 40])
@pytest.mark.parametrize("n", [33, 200])
def test_radius_past_thin_grids_matches_oracle(orc, dims, radius, n):
    rng = np.random.default_rng(n + radius)
    cell = 0.25
    pos = np.ones((n, 4), np.float32)
    # Some outside the grid too: they belong to its border cells.
    pos[:, :3] = rng.uniform(-0.3, np.asarray(dims) * cell + 0.3, (n, 3))
    got = _search(CudaBackend(), pos, dims, cell, radius * cell)
    want = _search(OracleBackend(), pos, dims, cell, radius * cell)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


def test_walk_costs_the_rows_of_the_grid():
    """641,601 rows of a radius of 400 cells, one of them inside the grid."""
    B, dims, cell = CudaBackend(), (400, 1, 1), 0.25
    pos = np.ones((64, 4), np.float32)
    pos[:, :3] = np.random.default_rng(5).uniform(0.0, np.asarray(dims) * cell, (64, 3))

    def fastest(h):
        took = []
        for _ in range(8):
            t0 = time.perf_counter()
            _search(B, pos, dims, cell, h)
            took.append(time.perf_counter() - t0)
        return min(took)

    fastest(cell)
    assert fastest(400 * cell) < 4.0 * fastest(cell)

"""Grids of two million cells and more around the four cells per bead at which
the cell sort changes from a thread per cell to a thread per bead: the lists
against the host's pairs, in the order of the cells and of the beads in them."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, Settings

pytestmark = pytest.mark.gpu

GRID = np.array([129, 127, 131])
CELLS = int(GRID.prod())
RADIUS = 0.45  # listed out to a radius and a skin radius: 1.1


def gas(n):
    """Free beads anywhere in the box, some of them six to a cell."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * GRID
    c = n // 600 * 6
    pos[:c] = np.floor(pos[:c:6]).repeat(6, axis=0) + rng.uniform(0.02, 0.98, (c, 3))
    pos = pos[rng.permutation(n)]
    st = Settings(dt=0.001, cutoff=1.0, box_unit_cell=1.0, box=tuple(map(float, GRID)), bc_type=0, skin_ratio=0.2)
    return g.chain_model(pos[:, None, :], st, ["A"], [PAIR_HS], [[50.0, 0, 0, 0]], radius=RADIUS)


def neighbours(pos, limit):
    """Ordered pairs nearer than the limit in cells that touch, with the rank of
    the partner's cell among the 27 (z, y, x ascending)."""
    p = cKDTree(np.mod(pos, GRID), boxsize=GRID).query_pairs(limit, output_type="ndarray")
    i, j = np.concatenate([p, p[:, ::-1]]).T
    cell = np.floor(pos).astype(np.int64)
    off = np.mod(cell[j] - cell[i] + 1, GRID)
    near = (off < 3).all(axis=1)
    rank = (off[:, 2] * 3 + off[:, 1]) * 3 + off[:, 0]
    i, j, rank = i[near], j[near], rank[near]
    o = np.lexsort((j, rank, i))
    return i[o], j[o]


@pytest.mark.parametrize("build", ["beads", "groups", "bricks"])
@pytest.mark.parametrize("n", [CELLS // 4, CELLS // 4 + 1, 300_001])
def test_order_and_pairs(n, build):
    from fibrenet_b200.native import Simulation
    m = gas(n)
    pos = np.asarray(m.pos)
    limit = float(np.float32(RADIUS)) + float(np.float32(float(np.float32(RADIUS)) + 0.2))
    want = neighbours(pos, limit)
    assert not set(zip(*neighbours(pos, limit + 1e-9))) ^ set(zip(*want))  # no pair is on the edge
    with Simulation(m, reorder=False, list_capacity=64) as s:
        assert s.lib.fn_n_cells(s.h) == CELLS
        s.set_list_build(build)
        s.rebuild()
        count, partners = s.lists()
        assert s.stats()["cell_overflow"] == 0 and s.stats()["list_overflow"] == 0
    i = np.repeat(np.arange(n), count)
    j = np.concatenate([partners[count > k, k] for k in range(count.max())])
    j = j[np.argsort(np.concatenate([np.flatnonzero(count > k) for k in range(count.max())]), kind="stable")]
    np.testing.assert_array_equal(i, want[0])
    np.testing.assert_array_equal(j, want[1])

"""List builds where a row of three cells holds more beads than one cell may
keep: the same lists as the build by bricks, with no cell, some cells and many
cells over their capacity, and as fast as with a capacity that no row reaches."""
import numpy as np
import pytest

from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, PAIR_LJ, Settings

pytestmark = pytest.mark.gpu


def gas(n, side, cell, mask=7, seed=1, radius=0.3, clump=0):
    """Pairs of beads anywhere in a box of side^3 cells, the first `clump` of
    them around two places, one of them at a periodic corner."""
    rng = np.random.default_rng(seed)
    box = np.full(3, side * cell)
    img = np.repeat(rng.uniform(0.0, 1.0, (n // 2, 1, 3)) * box, 2, axis=1)
    at = np.where(np.arange(clump)[:, None] % 2, 0.02 * cell, 1.5 * cell)
    img[:clump] = np.mod(at + rng.normal(0.0, 0.2 * cell, (clump, 3)), box)[:, None]
    img[:, 1, 0] = np.where(img[:, 0, 0] > 0.5 * box[0], img[:, 0, 0] - 0.5, img[:, 0, 0] + 0.5)
    st = Settings(dt=1e-7, cutoff=cell, box_unit_cell=cell, box=tuple(box), wall_k=1.0, bc_type=0 if mask == 7 else 1,
                  periodic_mask=mask)
    kinds = ([PAIR_HS, PAIR_LJ, PAIR_HS], [[50.0, 0, 0, 0], [1e-9, 1e-9, 0.5 * cell, 0], [50.0, 0, 0, 0]])
    return g.chain_model(img, st, ["A", "B"], *kinds, bead_type=np.arange(img.shape[0] * 2) % 2, radius=radius)


def lists(m, build, cap):
    from fibrenet_b200.native import Simulation
    with Simulation(m, list_capacity=128, cell_capacity=cap) as s:
        s.set_list_build(build)
        s.rebuild()
        st = s.stats()
        return (*s.lists(), st["cell_overflow"], st["list_overflow"])


# capacities: rows above it but no cell, a few cells, most cells, rows far above
# three of it; the last sizes on either side of the one up to which the default
# build takes four lanes per bead
@pytest.mark.parametrize("mask", [7, 2])
@pytest.mark.parametrize("n,side,cap,clump", [(4096, 8, 24, 0), (4096, 8, 12, 0), (4096, 8, 3, 0), (4096, 8, 24, 300),
                                              (4096, 8, 1, 300), (600, 3, 24, 0), (600, 4, 40, 200),
                                              (200_102, 29, 20, 0), (200_102, 29, 9, 200), (196_000, 29, 9, 200)])
def test_same_lists(n, side, cap, clump, mask):
    m = gas(n, side, 1.2, mask, clump=clump)
    want = lists(m, "bricks", cap)
    assert want[0].sum() > 0
    for build in ("beads", "groups"):
        for a, b in zip(lists(m, build, cap), want):
            np.testing.assert_array_equal(a, b, err_msg=build)


def rebuild_ms(m, build, cap):
    from fibrenet_b200.native import Simulation
    with Simulation(m, list_capacity=96, cell_capacity=cap) as s:
        s.set_list_build(build)
        s.enable_timing(True)
        best = np.inf
        for _ in range(6):
            s.step(80)
            best = min(best, s.kernel_time()["rebuild_ms"])
        return best


# eight beads per cell: nearly every bead has a row of more than 26, nearly no
# cell has
@pytest.mark.parametrize("build", ["beads", "groups"])
@pytest.mark.parametrize("n,side", [(21_952, 14), (314_432, 34)])
def test_capacity_of_long_rows_costs_no_time(n, side, build):
    m = gas(n, side, 1.8, seed=3)
    assert rebuild_ms(m, build, 26) < 1.4 * rebuild_ms(m, build, 256)


# networks of three cells a side (folded separations) and of eight in one
# context, below and above the size of the four-lane default
@pytest.mark.parametrize("n", [2000, 101_000])
def test_batch_of_short_and_long_boxes(n):
    ms = [gas(600, 3, 1.2, seed=5), gas(n, round((n / 8) ** (1 / 3)), 1.2, seed=6), gas(800, 4, 1.2, mask=2, seed=7),
          gas(n + 50, round((n / 6) ** (1 / 3)), 1.2, seed=8)]
    want = lists(ms, "bricks", 16)
    for build in ("beads", "groups"):
        for a, b in zip(lists(ms, build, 16), want):
            np.testing.assert_array_equal(a, b, err_msg=build)

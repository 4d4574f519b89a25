"""Grids of two million cells and more, where the scan takes eight cells per
thread and, with few beads in them, the cell sort one thread per bead: against
the oracle's MIRROR mode, bit for bit, cells over their capacity included."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, Settings

pytestmark = pytest.mark.gpu


def clusters(box, n, per, seed):
    """Free beads in tight clusters, some across the periodic sides."""
    rng = np.random.default_rng(seed)
    at = rng.uniform(0.0, 1.0, (n // per, 1, 3)) * box
    at[:4] = np.array([[0.1, 0.1, 0.1], [0.1, 0.1, box[2] - 0.1], [box[0] - 0.2, 5.0, 5.0], [5.0, 0.05, 7.0]])[:, None]
    pos = np.mod(at + rng.normal(0.0, 0.4, (n // per, per, 3)), box)
    pos = pos.reshape(-1, 1, 3)
    st = Settings(dt=0.001, cutoff=1.0, box_unit_cell=1.0, box=tuple(box), bc_type=0)
    return g.chain_model(pos, st, ["A"], [PAIR_HS], [[50.0, 0, 0, 0]])


# 2,146,173 cells (no multiple of eight) and one cell above 2^21
@pytest.mark.parametrize("box,n,per,cap", [((129.0, 127.0, 131.0), 6000, 6, 16), ((129.0, 127.0, 131.0), 6000, 6, 2),
                                           ((2097153.0 / 9.0, 3.0, 3.0), 3000, 5, 16)])
def test_sparse_grid(oracle_built, box, n, per, cap):
    from fibrenet_b200.native import Simulation
    m = clusters(np.array(box), n, per, 3)
    with Simulation(m, reorder=False, cell_capacity=cap, list_capacity=64) as s:
        assert s.lib.fn_n_cells(s.h) >= 2 << 20
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=cap, list_cap=64)
        s.step(17)
        o.run(17)
        for f in ("img", "force", "vel_old"):
            np.testing.assert_array_equal(s.get(f), o.get(f), err_msg=f)
        assert (s.stats()["cell_overflow"] > 0) == (cap == 2)

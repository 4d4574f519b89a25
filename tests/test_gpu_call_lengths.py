"""State after calls of every length around the rebuild interval (8): the call's
last step may stand alone in its segment.  Bit for bit against the mirror."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from gpu_util import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 10, 17])
def test_state_after_a_call_of_n_steps(oracle_built, n, graphs):
    from fibrenet_b200.native import Simulation
    m = g.plain_network(seed=4, fibres=9, beads=11, box=(16.0, 16.0, 6.0), z_range=(1.0, 5.0))
    m.vel = m.vel_old = np.random.default_rng(1).normal(0.0, 0.3, m.vel.shape).astype(np.float32).astype(np.float64)
    with Simulation(m, reorder=False, use_graphs=graphs) as s:
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=64, list_cap=64)
        for _ in range(2):
            s.step(n)
            o.run(n)
            for f in FIELDS:
                np.testing.assert_array_equal(s.get(f), o.get(f), err_msg=f)

"""Force terms with infinite coefficients against the oracle's MIRROR mode: the
infinities and the NaN that the plain operators give."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, Settings

pytestmark = pytest.mark.gpu


def bent_fibres(k_a):
    """Four fibres of three and more beads, each bent a little differently."""
    rng = np.random.default_rng(11)
    img = np.zeros((4, 6, 3))
    img[:, :, 0] = 4.0 + np.arange(6)
    img[:, :, 1] = (3.0 + 3.0 * np.arange(4))[:, None]
    img[:, :, 2] = 8.0
    img += rng.uniform(-0.2, 0.2, img.shape)
    st = Settings(dt=0.001, cutoff=1.0, box_unit_cell=1.0, box=(16.0, 16.0, 16.0), bc_type=0)
    return g.chain_model(img, st, ["A"], [PAIR_HS], [[50.0, 0, 0, 0]], k_s=100.0, k_a=k_a)


@pytest.mark.parametrize("kw", [{}, {"block_size": 64}, {"chain": False}])
def test_infinite_angle_stiffness(oracle_built, kw):
    from fibrenet_b200.native import Simulation
    m = bent_fibres(np.inf)
    with Simulation(m, reorder=False, list_capacity=64, **kw) as s:
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=64, list_cap=64)
        s.step(1)
        o.run(1)
        assert np.isinf(o.get("force")).sum() > 8
        for f in ("force", "vel_old"):
            np.testing.assert_array_equal(s.get(f), o.get(f), err_msg=f)

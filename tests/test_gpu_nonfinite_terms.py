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


# a radius that is not a number is near no other: the list builds that test in
# FP32 first against the build by bricks, which tests in FP64
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("later", [False, True])
@pytest.mark.parametrize("host", [False, True])
def test_lists_with_a_radius_or_skin_that_is_no_number(host, later, value):
    from fibrenet_b200.native import Simulation
    rng = np.random.default_rng(5)
    st = Settings(dt=0.001, cutoff=1.0, box_unit_cell=2.0, box=(12.0, 14.0, 16.0), bc_type=0)
    m = g.chain_model(rng.uniform(0.0, 12.0, (2000, 1, 3)), st, ["A"], [PAIR_HS], [[50.0, 0, 0, 0]], radius=0.5)
    odd = np.arange(0, m.n_beads, 50)
    skin = np.full(m.n_beads, 0.8)
    if later:
        skin[odd] = value
    else:
        m.radius[odd] = value
    got = []
    for build in ("bricks", "beads", "groups"):
        with Simulation(m, list_capacity=256, host_upload=host) as s:
            s.set_list_build(build)
            if later:
                s.set_skin(skin)
            s.rebuild()
            got.append(s.lists())
    assert later is False or np.isinf(value) or got[0][0].sum() > 0
    for c, p in got[1:]:
        np.testing.assert_array_equal(c, got[0][0])
        np.testing.assert_array_equal(p, got[0][1])

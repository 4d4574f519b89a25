"""The chain step of small contexts (five warps per up to 28 beads, contacts 16 at
a time) against the oracle's MIRROR mode, bit for bit: parts of a tile that end
within a fibre, single beads, lists of more than one round, and the same
networks with a block size given, which keeps one thread per bead."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from gpu_util import FIELDS

pytestmark = pytest.mark.gpu


def check(m, steps, lists=None, **kw):
    from fibrenet_b200.native import Simulation
    with Simulation(m, reorder=False, list_capacity=64, **kw) as s:
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=64, list_cap=64)
        for n in steps:
            s.step(n)
            o.run(n)
            for f in FIELDS:
                np.testing.assert_array_equal(s.get(f), o.get(f), err_msg=f)
        for a, b in zip(s.status(), o.status()):
            np.testing.assert_array_equal(a, b)
        if lists is not None:
            assert s.lists()[0].max() > lists


# tiles of 124 beads in five parts of 25
@pytest.mark.parametrize("block", [0, 128])
@pytest.mark.parametrize("beads,fibres", [(1, 1), (24, 1), (25, 1), (26, 1), (50, 1), (51, 1), (101, 1), (124, 1),
                                          (125, 1), (149, 1), (31, 9)])
def test_parts(oracle_built, beads, fibres, block):
    side = max(beads + 4.0, 8.0)
    m = g.plain_network(seed=beads, fibres=fibres, beads=beads, box=(side, side, 6.0), z_range=(1.0, 5.0))
    m.vel = m.vel_old = np.random.default_rng(2).normal(0.0, 0.3, m.vel.shape).astype(np.float32).astype(np.float64)
    check(m, [2, 9], block_size=block)


# contacts per bead below, at and above one and two rounds
@pytest.mark.parametrize("side,least", [(9.0, 12), (7.2, 17), (5.6, 33)])
def test_rounds_of_contacts(oracle_built, side, least):
    check(g.dense_mat(seed=3, fibres=50, beads=20, box=(side, side, side)), [3, 10], lists=least)


def test_damped_batch_of_several_laws(oracle_built):
    from fibrenet_b200.native import Simulation
    ms = [g.plain_network(seed=k, fibres=5 + k, beads=17, box=(22.0, 22.0, 6.0), z_range=(1.0, 5.0),
                          k_contact=50.0 + k) for k in range(4)]
    for m in ms:
        m.settings.damping = 0.3
    with Simulation(ms, list_capacity=64) as s, Simulation(ms, list_capacity=64, block_size=64) as t:
        for n in (1, 10, 7):
            s.step(n)
            t.step(n)
            for f in FIELDS:
                np.testing.assert_array_equal(s.get(f), t.get(f), err_msg=f)

"""The step sequence's kernels are placed before their predecessors end and wait
on the device.  Runs whose calls follow each other without a wait on the host,
in several contexts at once, equal the same runs synchronised call by call."""
import numpy as np
import pytest

from fibrenet_b200 import generate as g
from gpu_util import FIELDS

pytestmark = pytest.mark.gpu


def models():
    out = [g.plain_network(seed=3, fibres=1, beads=2, box=(8.0, 8.0, 8.0), z_range=(3.0, 5.0)),
           g.plain_network(seed=4, fibres=60, beads=31, box=(40.0, 40.0, 8.0), z_range=(1.0, 7.0)),
           g.dense_mat(seed=5, fibres=300, beads=40, box=(24.0, 24.0, 24.0))]
    rng = np.random.default_rng(0)
    for m in out:
        m.vel = m.vel_old = rng.normal(0.0, 0.2, m.vel.shape)
    return out


def run(m, sims, sync):
    rows = []
    for n in (1, 9, 16, 3):
        for s in sims:
            s.step(n)
            if sync:
                s.sync()
        for s in sims:
            s.rebuild()
            if sync:
                s.sync()
    for s in sims:
        rows.append(s.step_series(12, 5, energy=True))
    return rows


@pytest.mark.parametrize("kw", [{}, {"use_graphs": True}, {"chain": False}, {"list_capacity": 32, "block_size": 64}])
def test_unsynchronised_calls_equal_synchronised_ones(kw):
    from fibrenet_b200.native import Simulation
    got = []
    for sync in (True, False):
        sims = [Simulation(m, **kw) for m in models()]
        rows = run(None, sims, sync)
        got.append((rows, [{f: s.get(f) for f in FIELDS} for s in sims], [s.lists() for s in sims]))
        for s in sims:
            s.close()
    for a, b in zip(got[0][0], got[1][0]):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(got[0][1], got[1][1]):
        for f in FIELDS:
            np.testing.assert_array_equal(a[f], b[f], err_msg=f)
    for a, b in zip(got[0][2], got[1][2]):
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])


def test_displacement_mode():
    from fibrenet_b200.native import Simulation
    m = g.tensile_network(seed=2, fibres=60, beads=20, box=(66.0, 66.0, 20.0), clamp_hi=64.0, cell=3.0)
    m.vel = m.vel_old = np.random.default_rng(1).normal(0.0, 3.0, m.vel.shape) * (m.mass > 0)[:, None]
    got = []
    for sync in (True, False):
        with Simulation(m, verlet_skin=0.4) as s:
            for _ in range(40):
                s.step(5)
                if sync:
                    s.sync()
            got.append((s.get("img"), s.get("force"), s.lists(), s.stats()["rebuilds"]))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    np.testing.assert_array_equal(got[0][2][1], got[1][2][1])
    assert got[0][3] == got[1][3] and 1 < got[0][3] < 200

"""The step kernels' two ways of reading a network's constants (one pair law
for all bead types: as kernel parameters; several laws or networks: from
tables) and the shared-seed roots and quotients, against the oracle's MIRROR
mode, which uses the plain operators.  Tolerance: none, every bit."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, PAIR_HSR, PAIR_LJ, PAIR_ST, SPRING_HR_FL, Settings
from gpu_util import FIELDS

pytestmark = pytest.mark.gpu

LAWS = {"lj": (PAIR_LJ, [1.0, 1.0, 1.5, 0.0]), "hs": (PAIR_HS, [50.0, 0, 0, 0]),
        "st": (PAIR_ST, [5.0, 20.0, 1.0, 1.4]), "hsr": (PAIR_HSR, [50.0, 10.0, 1.2, 0])}


def network(law, uniform, beads, fibres, fail=False):
    """Parallel fibres a little under a bead apart (straight, unit spacing:
    squared lengths a rounding away from 1), two bead types; the second
    type's law differs in its strength unless `uniform`."""
    rng = np.random.default_rng(beads * 100 + fibres)
    side = beads + 6.0
    img = np.zeros((fibres, beads, 3))
    img[:, :, 0] = 3.0 + np.arange(beads)
    img[:, :, 1] = (1.0 + 0.97 * (np.arange(fibres) % 4))[:, None]
    img[:, :, 2] = (1.0 + 0.97 * (np.arange(fibres) // 4))[:, None]
    st = Settings(dt=0.001, cutoff=1.5, box_unit_cell=1.5, box=(side, 8.0, 8.0), bc_type=0)
    kind, raw = LAWS[law]
    other = [raw[0], 2.0 * raw[1], *raw[2:]] if law != "hs" else [2.0 * raw[0], 0, 0, 0]
    pr = [raw, raw if uniform else other, raw]
    vel = rng.normal(0.0, 0.3, (fibres * beads, 3))
    m = g.chain_model(img, st, ["A", "B"], [kind] * 3, pr, bead_type=np.arange(fibres * beads) % 2, k_s=100.0,
                      k_a=10.0, vel=vel, **(dict(spring_type=SPRING_HR_FL, s_c1=1e3, s_c2=2.0) if fail else {}))
    return m


def equal_to_mirror(m, steps, **kw):
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


# tiles of 64 - 4 = 60 beads: one bead, a tile less one, exact, one more, two
# tiles and a remainder
@pytest.mark.parametrize("chain", [True, False])
@pytest.mark.parametrize("beads,fibres", [(1, 1), (2, 1), (3, 1), (59, 1), (60, 1), (61, 1), (31, 4), (60, 2)])
def test_tile_edges(oracle_built, beads, fibres, chain):
    equal_to_mirror(network("hs", True, beads, fibres), [1, 9], block_size=64, chain=chain)


@pytest.mark.parametrize("chain", [True, False])
@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("law", sorted(LAWS))
def test_laws_uniform_and_tabled(oracle_built, law, uniform, chain):
    equal_to_mirror(network(law, uniform, 33, 7, fail=True), [30], chain=chain)


@pytest.mark.parametrize("law", ["hs", "hsr", "lj"])
@pytest.mark.parametrize("gap", [1e-35, 1e-20, 3e-7])
def test_distances_outside_the_shared_seed_range(oracle_built, law, gap):
    """Beads closer than the shared-seed arithmetic takes (and one pair inside
    its range), spring ends included, fall back to the operators."""
    kind, raw = LAWS[law]
    st = Settings(dt=1e-9, cutoff=1.5, box_unit_cell=1.5, box=(6.0, 6.0, 6.0), bc_type=0)
    z = (0.0, 0.0, 0.0)
    beads = [(0, i, 0, 0.5, 0.0, p, z, p) for i, p in
             enumerate([(0.0, 0.0, 0.0), (gap, 0.0, 0.0), (0.0, 2 * gap, gap), (3.0, 3.0, 3.0), (3.0, 4.1, 3.0)])]
    m = g.explicit_model(st, ["A"], {(0, 0): (kind, raw)}, beads,
                         springs=[(0, 0, 0, 1, 1.0, 10.0, 0.0, 0.0), (0, 0, 3, 4, 1.0, 10.0, 0.0, 0.0)])
    if law == "lj":
        # the overlapping pairs' force is beyond FP32: keep one within range
        m.pos[1] = m.img[1] = (0.6, 0.0, 0.0)
        m.pos[2] = m.img[2] = (0.0, 0.7, gap)
    equal_to_mirror(m, [2])


# both chain kernels that read networks' settings from tables and the one pair
# law from the kernel parameters: by default the small-context form, with a
# block size one thread per bead
@pytest.mark.parametrize("block", [0, 64])
@pytest.mark.parametrize("law", sorted(LAWS))
def test_networks_of_one_law(oracle_built, law, block):
    from fibrenet_b200.native import Simulation
    ms = [network(law, True, beads, fibres) for beads, fibres in ((33, 3), (1, 5), (60, 2))]
    for k, m in enumerate(ms):
        m.settings.damping = 0.1 * k
    with Simulation(ms, reorder=False, list_capacity=64, block_size=block) as s:
        s.step(1)
        s.step(11)
        got = {f: s.get(f) for f in FIELDS}
    first = 0
    for m in ms:
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=64, list_cap=64)
        o.run(1)
        o.run(11)
        n = len(o.get("pos"))
        for f in FIELDS:
            np.testing.assert_array_equal(got[f][first:first + n], o.get(f), err_msg=f)
        first += n

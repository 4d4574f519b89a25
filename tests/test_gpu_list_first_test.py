"""The list builds that test candidates in FP32 first (one thread, four and
eight lanes per bead) against the build by bricks, which tests every candidate
in FP64: the same lists, entry for entry.  Also against the oracle's MIRROR
mode on small networks."""
import numpy as np
import pytest

import pyoracle as po
from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, PAIR_HSR, PAIR_LJ, PAIR_ST, Settings

pytestmark = pytest.mark.gpu

LAWS = {"lj": (PAIR_LJ, [1.0, 1.0, 1.0, 0.0]), "hs": (PAIR_HS, [50.0, 0, 0, 0]),
        "st": (PAIR_ST, [5.0, 20.0, 1.0, 1.0]), "hsr": (PAIR_HSR, [50.0, 10.0, 0.9, 0])}


def gas(n, box, law, mask, seed=1, radii=(0.5, 0.5), two_laws=False):
    """Short free fibres (pairs of beads) anywhere in the box."""
    rng = np.random.default_rng(seed)
    img = np.repeat(rng.uniform(0.0, 1.0, (n // 2, 1, 3)) * box, 2, axis=1)
    img[:, 1, 0] = np.where(img[:, 0, 0] > 0.5 * box[0], img[:, 0, 0] - 0.7, img[:, 0, 0] + 0.7)
    st = Settings(dt=1e-5, cutoff=1.0, box_unit_cell=1.0, box=tuple(float(b) for b in box), wall_k=1.0,
                  bc_type=0 if mask == 7 else 1, periodic_mask=mask)
    kinds = [LAWS[law][0]] * 3
    raws = [LAWS[law][1]] * 3
    if two_laws:
        kinds[1], raws[1] = LAWS["hs" if law != "hs" else "lj"]
    N = img.shape[0] * 2
    return g.chain_model(img, st, ["A", "B"], kinds, raws, bead_type=np.arange(N) % 2,
                         radius=rng.uniform(*radii, N))


def lists(m, build, **kw):
    from fibrenet_b200.native import Simulation
    with Simulation(m, list_capacity=64, **kw) as s:
        s.set_list_build(build)
        s.rebuild()
        c, p = s.lists()
        st = s.stats()
        return c, p, st["cell_overflow"], st["list_overflow"]


def same(m, **kw):
    want = lists(m, "bricks", **kw)
    for build in ("beads", "groups"):
        got = lists(m, build, **kw)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b, err_msg=build)
    return want


# grids of 3, 4 and 5 cells (too small for the FP32 test, for its inner radius,
# and for neither), with and without periodic sides
@pytest.mark.parametrize("mask", [0, 2, 5, 7])
@pytest.mark.parametrize("box", [(3.0, 3.0, 3.0), (4.2, 3.5, 5.9), (9.3, 5.0, 40.7), (1000.0, 3.3, 12.0)])
def test_small_grids(box, mask):
    m = gas(int(min(box[0] * box[1] * box[2], 4000)) // 2 * 2, np.array(box), "hs", mask)
    assert same(m)[0].sum() > 0


@pytest.mark.parametrize("two_laws", [False, True])
@pytest.mark.parametrize("law", sorted(LAWS))
def test_laws_and_radii(law, two_laws):
    same(gas(3000, np.array([14.0, 15.0, 16.0]), law, 7, radii=(0.2, 0.5), two_laws=two_laws))


def test_skin_set_later():
    from fibrenet_b200.native import Simulation
    m = gas(2000, np.array([12.0, 13.0, 14.0]), "hs", 7)
    got = []
    for build in ("bricks", "beads", "groups"):
        with Simulation(m, list_capacity=64, use_graphs=True) as s:
            s.set_list_build(build)
            s.step(9)
            s.set_skin(np.linspace(0.3, 0.45, m.n_beads))
            s.step(9)
            got.append(s.lists())
    for c, p in got[1:]:
        np.testing.assert_array_equal(c, got[0][0])
        np.testing.assert_array_equal(p, got[0][1])


# more near candidates than a thread or group keeps, cells over their capacity
@pytest.mark.parametrize("cap", [1, 6, 64])
def test_crowded_cells(cap):
    assert same(gas(1500, np.array([5.0, 6.0, 7.0]), "hs", 7), cell_capacity=cap)[0].max() > 32 or cap < 64


# above the size up to which the default build takes four lanes per bead
@pytest.mark.parametrize("box,mask", [((3.2, 250.0, 260.0), 7), ((60.0, 61.0, 62.0), 7), ((60.0, 61.0, 62.0), 2)])
def test_one_thread_per_bead(box, mask):
    same(gas(200_102, np.array(box), "hsr", mask))


@pytest.mark.parametrize("law", sorted(LAWS))
def test_lists_of_the_mirror(oracle_built, law):
    m = gas(900, np.array([9.0, 10.0, 11.0]), law, 7)
    from fibrenet_b200.native import Simulation
    with Simulation(m, reorder=False, list_capacity=64) as s:
        o = po.OracleSim(m, po.MODE_MIRROR, cell_cap=64, list_cap=64)
        s.step(17)
        o.run(17)
        np.testing.assert_array_equal(s.get("img"), o.get("img"))
        np.testing.assert_array_equal(s.get("force"), o.get("force"))

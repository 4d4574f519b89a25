"""The contact energy of beads that coincide: not finite for the
Lennard-Jones law, whose potential is singular there; that of the overlap for
the penalty law."""
import numpy as np
import pytest

from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, PAIR_LJ, Settings

pytestmark = pytest.mark.gpu


def contact_energy(law, gap):
    from fibrenet_b200.native import Simulation
    st = Settings(dt=0.001, cutoff=2.0, box_unit_cell=2.0, box=(8.0, 8.0, 8.0), bc_type=0)
    at = [(3.0, 3.0, 3.0), (3.0 + gap, 3.0, 3.0)]
    beads = [(0, i, 0, 0.5, 1.0, p, (0.0, 0.0, 0.0), p) for i, p in enumerate(at)]
    with Simulation(g.explicit_model(st, ["A"], {(0, 0): law}, beads), list_capacity=64) as s:
        s.rebuild()
        e = s.energy(0)
        assert e["contacts"] == 1
        return e["contact"]


def test_lennard_jones():
    law = (PAIR_LJ, [1.0, 1.0, 1.5])
    assert np.isfinite(contact_energy(law, 1e-3))
    assert not np.isfinite(contact_energy(law, 0.0))


def test_penalty():
    assert contact_energy((PAIR_HS, [50.0]), 0.0) == 0.5 * 50.0 * 1.0

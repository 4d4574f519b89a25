"""fn_download into pageable and pinned arrays, below and above the size from
which a pageable destination's pages are touched beforehand.  Tolerance: none."""
import ctypes as C

import numpy as np
import pytest
import torch

from fibrenet_b200 import generate as g
from fibrenet_b200.native import FIELDS, Simulation

pytestmark = pytest.mark.gpu


# 24 bytes per bead: 16 MB are 699,051 beads
@pytest.mark.parametrize("fibres,beads", [(27, 37), (10001, 70)])
def test_pageable_and_pinned(fibres, beads):
    side = np.sqrt(fibres / 200.0) * 100.0
    m = g.plain_network(seed=6, fibres=fibres, beads=beads, box=(side, side, 10.0))
    with Simulation(m) as s:
        s.step(2)
        view = s.get("force")
        pinned = torch.empty((s.nb, 3), dtype=torch.float64).pin_memory()
        assert s.lib.fn_download(s.h, FIELDS["force"], C.cast(pinned.data_ptr(), C.POINTER(C.c_double))) == 0
        np.testing.assert_array_equal(pinned.numpy(), view)
        assert np.abs(view).max() > 0.0

"""fn_download against the device array itself, below and above the size from
which missing pages of the destination are faulted in first: a fresh array, the
same array again, and one half of whose pages are there.  Tolerance: none."""
import ctypes as C
import mmap

import numpy as np
import pytest
import torch

from fibrenet_b200 import generate as g
from fibrenet_b200.native import FIELDS, Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fibres,beads", [(27, 37), (10001, 70)])
def test_against_the_device_array(fibres, beads):
    side = np.sqrt(fibres / 200.0) * 100.0
    m = g.plain_network(seed=6, fibres=fibres, beads=beads, box=(side, side, 10.0))
    with Simulation(m) as s:
        s.step(2)
        for field in ("img", "force"):
            device = torch.as_tensor(s.device_view(field), device="cuda")[:, :3].double().cpu().numpy()
            want = np.empty_like(device)
            want[s.permutation()] = device
            assert np.abs(want).max() > 0.0
            fresh = mmap.mmap(-1, 24 * s.nb)
            half = mmap.mmap(-1, 24 * s.nb)
            half[:12 * s.nb] = b"\1" * (12 * s.nb)
            for buffer in (fresh, fresh, half):
                out = np.frombuffer(buffer, np.float64).reshape(s.nb, 3)
                assert s.lib.fn_download(s.h, FIELDS[field], C.cast(out.ctypes.data, C.POINTER(C.c_double))) == 0
                np.testing.assert_array_equal(out, want)

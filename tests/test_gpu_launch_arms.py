"""The kernels of a step, a rebuild and an adjoint sweep are placed before their
predecessors end and wait on the device.  The same runs with every launch
waited for on the host (CUDA_LAUNCH_BLOCKING), where no two kernels overlap,
give every bit of state, lists, observables and gradients, on networks of one
and of several waves of blocks."""
import os
import subprocess
import sys

import numpy as np
import pytest

from launch_arms import CASES

pytestmark = pytest.mark.gpu

PROGRAM = os.path.join(os.path.dirname(os.path.abspath(__file__)), "launch_arms.py")


@pytest.mark.parametrize("case", sorted(CASES))
def test_overlapped_equals_one_by_one(case, tmp_path):
    got = []
    for blocking in ("0", "1"):
        out = str(tmp_path / f"{blocking}.npz")
        p = subprocess.run([sys.executable, PROGRAM, case, out], env={**os.environ, "CUDA_LAUNCH_BLOCKING": blocking},
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-3000:]
        with np.load(out) as f:
            got.append({k: f[k] for k in f.files})
    assert got[0].keys() == got[1].keys()
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
    assert got[0]["count"].sum() > 0 and np.abs(got[0]["force"]).max() > 0.0

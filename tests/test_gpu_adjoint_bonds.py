"""Adjoint bond and bead kernels at bond counts around their blocks of 128
(each block's last threads, a last block of one thread), both bond paths,
against the FP64 torch reference.  Tolerance: 1e-3 norm-wise, the bound of the
device's FP32 adjoint state (as for the larger network of the adjoint tests)."""
import numpy as np
import pytest

from test_adjoint import gpu_grads, pull, ref_grads, rel

pytestmark = pytest.mark.gpu


# fibres x (beads - 1 springs + beads - 2 angles): 129, 255, 513
@pytest.mark.parametrize("chain", [True, False])
@pytest.mark.parametrize("seed,fibres,beads,bonds", [(11, 3, 23, 129), (14, 15, 10, 255), (11, 27, 11, 513)])
def test_bond_counts(seed, fibres, beads, bonds, chain):
    m = pull(seed=seed, fibres=fibres, beads=beads)
    assert len(m.s_type) + len(m.a_k) == bonds
    w = np.random.default_rng(3).normal(size=(4, 1, 3))
    _, got = gpu_grads(m, 4, 10, 20, w, chain=chain)
    _, ref = ref_grads(m, 4, 10, w[:, 0, :])
    for k in ref:
        assert np.linalg.norm(ref[k]) > 0, k
        assert rel(got[k], ref[k]) < 1e-3, (k, rel(got[k], ref[k]))

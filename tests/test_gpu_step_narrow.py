"""The chain step with one thread per bead on small networks, at block sizes
around the default's (which there is the form with five warps per 28 beads),
against the oracle's MIRROR mode: tiles of 92 and 188 beads, one less, exact
and one more, and two tiles with a remainder."""
import pytest

from test_gpu_step_constants import equal_to_mirror, network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,beads,fibres", [(96, 91, 1), (96, 92, 1), (96, 93, 1), (96, 31, 9), (192, 187, 1),
                                                (192, 188, 1), (192, 189, 1), (192, 47, 9)])
def test_tile_edges(oracle_built, block, beads, fibres):
    equal_to_mirror(network("lj", False, beads, fibres), [1, 9], block_size=block)

"""Surrogate layers whose operands come by TMA, at the shapes of their tiles and rings: a second tile
of 64 or 96 pixels a row (128- and 64-byte boxes), enough tiles that every ring slot is used again,
with one and with two tiles a row.  FP64 oracle, the bounds of the BF16 network (forward 3e-2, each
parameter group's gradient 6e-2)."""
import pytest

from test_gpu_fno_edges import test_forward_and_gradients as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B", [(224, 1), (192, 9), (96, 30)])
def test_rings_and_partial_tiles(S, B):
    _check(S, B)

"""Surrogate gradients at the sizes where the fused backward kernels change shape: one slice pair a
sample and one sample (fewer slices than blocks), sides that are no multiple of the 128-pixel tile,
two tiles a pixel row, and a batch with several slices per block.  FP64 oracle, the bounds of the
BF16 network (forward 3e-2, each parameter group's gradient 6e-2)."""
import numpy as np
import pytest

from oracle import fno_oracle as O
from test_gpu_fno import FWD_TOL, GRAD_TOL, _groups, _net, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B", [(32, 1), (96, 2), (160, 1), (256, 1), (64, 40)])
def test_forward_and_gradients(S, B):
    torch = pytest.importorskip("torch")
    net, p = _net(S, B, seed=3 + S)
    rng = np.random.default_rng(S + B)
    x = rng.standard_normal((B, 6, S, S)).astype(np.float32)
    dy = rng.standard_normal((B, S, S)).astype(np.float32)
    y = net.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    net.backward(torch.from_numpy(dy).cuda())
    g = net.get_grads()
    net.backward(torch.from_numpy(dy).cuda())
    assert np.array_equal(g, net.get_grads())  # fixed summation order
    q, cache = O.forward(p, x)
    want = O.backward(p, cache, dy)
    assert _rel(y, q) < FWD_TOL
    for name, (a, b) in _groups().items():
        assert _rel(g[a:b], want[a:b]) < GRAD_TOL, (name, _rel(g[a:b], want[a:b]))
    net.close()

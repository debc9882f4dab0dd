"""A surrogate whose waits run out (a bound of 0 polls) reports it in the call where it happened; the
next call on the same handle, with the default bound, is exact again.  Sides on both of the DFT's paths
(one fused kernel up to 128, general products above), batches of few and of many blocks."""
import numpy as np
import pytest

from fastiso_b200 import abi
from fastiso_b200.fno import FNO, N_IN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B", [(32, 1), (96, 7), (128, 16), (160, 2)])
def test_handle_recovers_after_a_timeout(S, B):
    torch = pytest.importorskip("torch")
    lib = abi.load_library()
    g = torch.Generator(device="cpu").manual_seed(S + B)
    x = torch.randn(B, N_IN, S, S, generator=g).cuda()
    dy = torch.randn(B, S, S, generator=g).cuda()
    net = FNO(S, max_batch=B, seed=3)
    y = net.forward(x).clone()
    net.backward(dy)
    grads, params = net.get_grads(), net.get_params()
    for call in (lambda: net.forward(x), lambda: net.backward(dy), lambda: net.train_step(x, dy, 1e-3)):
        net.forward(x)
        assert lib.fi_debug_set_wait_limit(abi.FI_WAIT_TC_POLLS, 0) == abi.FI_OK
        try:
            with pytest.raises(abi.FiError) as e:
                call()
        finally:
            assert lib.fi_debug_set_wait_limit(abi.FI_WAIT_TC_POLLS, -1) == abi.FI_OK
        assert e.value.code == abi.FI_ERR_TIMEOUT
        with pytest.raises(abi.FiError) as e:  # no backward pass from a failed call's activations
            net.backward(dy)
        assert e.value.code == abi.FI_ERR_STATE
    assert np.array_equal(net.get_params(), params)  # no step from its gradients
    assert torch.equal(net.forward(x), y)
    net.backward(dy)
    assert np.array_equal(net.get_grads(), grads)
    net.train_step(x, dy, 1e-3)
    stepped = net.get_params()
    net.set_params(params)
    net.train_step(x, dy, 1e-3)
    assert np.array_equal(net.get_params(), stepped)  # the failed step was not counted
    net.close()

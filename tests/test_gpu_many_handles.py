"""A handle does not change what another one may launch: the shared-memory limit is a property of a
kernel on the device, so a small grid's handle made beside a large one's must leave it alone.  The
large handle's results are bitwise those of its run before the small one existed."""
import numpy as np
import pytest

import fastiso_b200 as F
from test_gpu_ensemble import member
from test_gpu_parity import small_sim

pytestmark = pytest.mark.gpu


def _rhs(sim, t):
    u = -40 * np.exp(-sim.domain.R**2 / (2 * (0.3 * sim.domain.Wx) ** 2))
    dudt = np.zeros_like(u)
    F.update_diagnostics(dudt, u, sim, t)
    return u, dudt


@pytest.mark.parametrize("small_form", ["fp64", "fp32"])
def test_fp64_form(small_form):
    alone = small_sim("fp64", 200, 150)
    want = [_rhs(alone, t) for t in (0.5, 12.5)]  # with and without the convolutions
    alone.close()
    sim = small_sim("fp64", 200, 150)
    got = [_rhs(sim, 0.5)]
    small = small_sim(small_form, 8, 8)
    _rhs(small, 0.5)
    got.append(_rhs(sim, 12.5))
    for (u, d), (uw, dw) in zip(got, want):
        assert np.array_equal(u, uw) and np.array_equal(d, dw)
    small.close()
    sim.close()


def test_persistent_kernel(monkeypatch):
    monkeypatch.setenv("FI_PERSIST_RESIDENT", "0")

    def run(beside):
        sim = small_sim("fp32", 130, 165)
        integ = F.init_integrator(sim)
        F.step(integ, 10.0)
        small = None
        if beside:
            small = small_sim("fp32", 8, 8)
            F.step(F.init_integrator(small), 10.0)
        F.step(integ, 10.0)
        u = sim.get_field("u")
        for s in (sim, small):
            if s:
                s.close()
        return u

    assert np.array_equal(run(False), run(True))


def test_ensembles():
    def run(beside):
        sims = [member(96, 21.0, 1), member(128, 20.5, 2)]
        for s in sims:
            F.init_integrator(s)
        ens = F.Ensemble(sims)
        assert ens.step(10.0) == [0, 0]
        other = []
        if beside:
            other = [member(16, 21.0, 3)]
            F.init_integrator(other[0])
            F.Ensemble(other).step(10.0)
        assert ens.step(10.0) == [0, 0]
        u = [s.get_field("u") for s in sims]
        for s in sims + other:
            s.close()
        return u

    for a, b in zip(run(False), run(True)):
        assert np.array_equal(a, b)

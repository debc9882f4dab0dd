"""Row-major field transfers (fi_get_field_rowmajor, fi_set_field_rowmajor, fi_rhs_rowmajor) against
the column-major ones: the same values whatever the caller's layout, at sides below, at and above
the 32-cell tile of the device's transposition."""
import numpy as np
import pytest

import fastiso_b200 as F
from fastiso_b200 import abi

pytestmark = pytest.mark.gpu


def _sim(form, nx, ny):
    domain = F.RegionalDomain(15e3 * nx, 15e3 * ny, nx, ny)
    x, y = domain.X / domain.Wx, domain.Y / domain.Wy
    eta = 10 ** (21 + 0.3 * np.sin(3 * x + y))
    se = F.SolidEarth(domain, layer_boundaries=[100e3], layer_viscosities=eta.reshape(nx, ny, 1))
    sim = F.Simulation(domain, F.BoundaryConditions(domain),
                       F.RegionalSeaLevel(surface=F.LaterallyVariableSeaSurface()), se, (0.0, 100.0), form=form)
    return sim, 1000.0 * np.clip(1 - x ** 2 - 2 * (y - 0.1) ** 2, 0, None)


@pytest.mark.parametrize("form", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(4, 5), (32, 64), (33, 31), (70, 45)])
def test_layouts_agree(form, nx, ny):
    out = []
    for order in "CF":
        sim, ice = _sim(form, nx, ny)
        integ = F.init_integrator(sim)
        sim.now.H_ice = np.array(ice, order=order)
        sim.now.u = np.array(-0.01 * ice, order=order)
        F.step(integ, 12.0)
        got = {f: sim.get_field(f) for f in ("u", "ue", "dudt", "dz_ss", "H_ice", "z_ss", "litho_rigidity")}
        for f, a in got.items():
            flat = np.empty(nx * ny)
            assert sim.lib.fi_get_field(sim._handle, abi.FIELDS[f], abi.dptr(flat), flat.size) == abi.FI_OK
            assert np.array_equal(a, abi.from_julia_layout(flat, nx, ny)), f
        assert np.array_equal(got["H_ice"], ice if form == "fp64" else ice.astype(np.float32))
        u, dudt = np.array(-0.02 * ice, order=order), np.zeros((nx, ny), order=order)
        F.update_diagnostics(dudt, u, sim, 13.0)
        got.update(rhs_u=u, rhs_dudt=dudt, now_u=sim.now.u, now_dudt=sim.now.dudt)
        assert np.array_equal(u, got["now_u"]) and np.array_equal(dudt, got["now_dudt"])
        out.append(got)
        sim.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]) and np.all(np.isfinite(out[0][f])), f


def test_wrong_sizes_stay_refused():
    sim, ice = _sim("fp32", 20, 24)
    sim.init_problem()
    for bad in (ice[:10], np.zeros(7), ice.T):
        if bad.size != ice.size:
            with pytest.raises(abi.FiError):
                sim.set_field("H_ice", bad)
    with pytest.raises(abi.FiError):
        sim.set_field("dudt", ice)
    sim.close()

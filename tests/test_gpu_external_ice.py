"""External ice and displacement in both layouts at the sizes around which the change of layout and the
ice's rounding to FP32 move from the host to the device (column-major 16384 cells, row-major 8192)."""
import numpy as np
import pytest

import fastiso_b200 as F
from fastiso_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(5, 7), (64, 128), (127, 65), (128, 128), (127, 129), (129, 128), (113, 145)])
def test_external_ice_layouts(form, nx, ny):
    domain = F.RegionalDomain(15e3 * nx, 15e3 * ny, nx, ny)
    se = F.SolidEarth(domain, layer_boundaries=[100e3], layer_viscosities=np.full((nx, ny, 1), 1e21))
    bcs = F.BoundaryConditions(domain, ice_thickness=F.ExternallyUpdatedIceThickness())
    sim = F.Simulation(domain, bcs, F.RegionalSeaLevel(), se, (0.0, 100.0), form=form)
    sim.init_problem()
    rng = np.random.default_rng(nx + ny)
    for order in "CF":
        ice = np.array(1000 * rng.random((nx, ny)), order=order)
        sim.set_field("H_ice", ice)
        flat = np.empty(nx * ny)
        assert sim.lib.fi_get_field(sim._handle, abi.FIELDS["H_ice"], abi.dptr(flat), flat.size) == abi.FI_OK
        want = ice if form == "fp64" else ice.astype(np.float32)
        assert np.array_equal(abi.from_julia_layout(flat, nx, ny), want)
        sim.set_field("u", -ice)
        if form == "fp32":  # the FP64 form reads u as of the last right-hand side
            assert np.array_equal(sim.get_field("u"), -ice)
    sim.close()

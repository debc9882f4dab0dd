"""The resident step kernel (a block keeps its row tile in shared memory) against k_persist:
the same arithmetic on the same elements in the same order, so the states are bitwise equal.
Sizes at the edges of its dispatch: the smallest grids, odd sides, factors without a register
butterfly, the compiled sequences, tiles enlarged to one per SM (more than 296 rows of height 2),
an odd number of rows there, column tasks enlarged (more than 296 columns of the half spectrum),
buffers that no longer fit (512 and wider)."""
import numpy as np
import pytest

import fastiso_b200 as F

pytestmark = pytest.mark.gpu


def _run(monkeypatch, resident, nx, ny, years, mask):
    monkeypatch.setenv("FI_PERSIST_RESIDENT", "1" if resident else "0")
    cell = 30e3
    domain = F.RegionalDomain(0.5 * cell * nx, 0.5 * cell * ny, nx, ny)
    rng = np.random.default_rng(100 * nx + ny)
    x, y = domain.X / domain.Wx, domain.Y / domain.Wy
    log_eta = 21 + 0.4 * np.sin(3 * x) * np.cos(2 * y) + 0.05 * rng.standard_normal((nx, ny))
    thick = 110e3 + 25e3 * np.cos(2.5 * x + y)
    ice = 1500.0 * np.clip(1 - 2 * (x - 0.1) ** 2 - 2 * y ** 2, 0, None)
    se = F.SolidEarth(domain, layer_boundaries=thick.reshape(nx, ny, 1),
                      layer_viscosities=(10 ** log_eta).reshape(nx, ny, 1),
                      maskactive=(x ** 2 + y ** 2 < 1.2) if mask else None)
    it = F.TimeInterpolatedIceThickness([0.0, 1.0, 500.0], [0 * ice, ice, 0.5 * ice], domain)
    sim = F.Simulation(domain, F.BoundaryConditions(domain, ice_thickness=it),
                       F.RegionalSeaLevel(surface=F.LaterallyVariableSeaSurface()), se, (0.0, 400.0), form="fp32",
                       u_ref=0.01 * thick / 1e3 if mask else None)
    integ = F.init_integrator(sim)
    for _ in range(2):
        F.step(integ, years)
    out = {f: sim.get_field(f) for f in ("u", "ue", "dudt", "dz_ss")}
    st = sim.stats()
    sim.close()
    return out, st


@pytest.mark.parametrize("nx,ny,years,mask", [
    (4, 4, 12.0, False), (5, 7, 12.0, False), (33, 24, 12.0, True), (64, 64, 12.0, False), (130, 165, 12.0, True),
    (96, 96, 12.0, False), (128, 128, 12.0, True), (192, 192, 12.0, False), (256, 256, 12.0, False),
    (40, 297, 6.0, False), (64, 298, 6.0, True), (597, 40, 6.0, False), (512, 512, 6.0, False), (1100, 64, 6.0, False),
])
def test_resident_bitwise(monkeypatch, nx, ny, years, mask):
    a, sa = _run(monkeypatch, True, nx, ny, years, mask)
    b, sb = _run(monkeypatch, False, nx, ny, years, mask)
    assert sa["naccept"] > 2 and sa["nsparse"] >= 1
    for k in ("naccept", "nreject", "nf", "nsparse"):
        assert sa[k] == sb[k], (k, sa[k], sb[k])
    for f in a:
        assert np.all(np.isfinite(a[f])) and np.array_equal(a[f], b[f]), (f, np.abs(a[f] - b[f]).max())

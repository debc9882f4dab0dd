"""The plain FP64 form's fused right-hand side against the FP64 oracle at the sizes where its
stencils and transforms can go wrong: the smallest grids (every cell at an edge), one row or column
more than an edge, odd sides with factors that have no register butterfly, more cells than one
pass of the grid-stride loops.  Tolerance: 1e-10 rel-L2, the form's per-right-hand-side bound."""
import numpy as np
import pytest

import fastiso_b200 as F
from helpers import F_, rel_l2
from test_gpu_parity import pair, small_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 4), (4, 7), (11, 13), (33, 26), (256, 31)])
def test_fused_rhs_matches_oracle(nx, ny):
    sim = small_sim("fp64", nx, ny, t_end=100.0)
    ref = pair(sim)
    rng = np.random.default_rng(nx + 100 * ny)
    u = -40 * np.exp(-sim.domain.R**2 / (2 * (0.3 * sim.domain.Wx) ** 2)) + 0.3 * rng.standard_normal((nx, ny))
    for t in (0.5, 12.5, 31.0):
        ug, dg = u.copy(), np.zeros_like(u)
        F.update_diagnostics(dg, ug, sim, t)
        _, dr = ref.rhs(t, F_(u))
        assert rel_l2(F_(dg), dr) < 1e-10, (t, rel_l2(F_(dg), dr))
        u = u + 0.1 * dg
    sim.close()
    ref.close()

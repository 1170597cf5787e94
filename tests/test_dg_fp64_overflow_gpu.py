"""FP64 DG right-hand sides whose fluxes overflow: NaN, infinities and finite
values where the oracle has them."""
import numpy as np
import pytest

from test_dg_fp64_tiles_gpu import open_solver, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [2, 3])
@pytest.mark.parametrize("var", [1, 2])  # F alone overflows, G alone
def test_flux_that_overflows_inside_a_cell(restatement, P, var):
    """A momentum of (P_0 - P_2)(xi) (P_0 - P_2)(eta): its square overflows at
    the cell's inner points and not on its faces, so the face integrals do not
    hide which of the volume terms are NaN."""
    c, d, b = problem(P, 12, 70, False, 9)
    d[:, 1:, 6, 33:36] = 0.0
    d[:3, 0, 6, 33:36] = np.array([1.0, 0.0, 0.0])[:, None]
    for px in (0, 2):
        for py in (0, 2):
            d[var, px * (P + 1) + py, 6, 34] = 1e160 * (-1) ** ((px + py) // 2)
    with open_solver(P, c, b, limiter="none") as s:
        s.set_state(d)
        out = s.rhs(0.0)
    with np.errstate(all="ignore"):
        ref = restatement.dg_rhs(P, d.copy(), b, c.da, c.gamma)[1]
    assert 0 < np.isnan(ref[var, :, 6, 34]).sum() < (P + 1) ** 2
    assert np.array_equal(out, ref, equal_nan=True)

"""The FP64_FMA path fuses multiply-adds; its quotients stay correctly rounded.

Supersonic flow to the right whose cells are all extrema: every MUSCL slope is
0, the flux through a face is the left cell's own, and its mass flux rho (m /
rho) is m exactly when m / rho, representable here, comes out exactly."""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp64_fma"])
def test_exact_quotients_come_out_exactly(precision):
    ny, nx = 12, 2000
    c = cases.four_quadrant(nx, seed=1, ny=ny)
    r = np.random.default_rng(5)
    j = np.arange(nx)
    rho = (r.integers(1 << 18, 1 << 19, nx) + (j % 2) * (5 << 17)) * 2.0 ** -19  # [0.5, 1), [1.75, 2.25)
    u = r.integers(8 << 18, 9 << 18, nx) * 2.0 ** -18
    m = rho * u
    assert np.array_equal(m / rho, u)
    U = np.zeros((4, ny, nx))
    U[0], U[1], U[3] = rho, m, 0.51 * m * u
    with Solver(method="weno", recon="muscl_minmod", precision=precision) as s:
        s.set_mesh(ny, nx, c.da, c.gamma, c.bctype)
        s.set_state(U)
        dU = s.rhs(c.da)[0]
    k = slice(6, nx - 6)
    assert np.array_equal(dU[6, k], (m[:-1] - m[1:])[5:nx - 7])

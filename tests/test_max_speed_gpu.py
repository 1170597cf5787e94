"""The CFL reductions at ragged widths: bit-equal to the oracle's.

The WENO reduction reads pairs of neighbouring cells, so odd widths end in
half a pair, and both walk pitched rows, so widths just below, at and above a
multiple of 32 cells have most, none and one of their padding columns.  The
random perturbation puts the maximum anywhere; the spike puts it in the last
column.  The reduction is exact (a max of identically rounded values), so the
comparison is equality.
"""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver, cases

pytestmark = pytest.mark.gpu

SIZES = [(7, 7), (9, 31), (8, 32), (11, 33), (300, 65), (257, 1030)]


def state(ny, nx, nm, seed):
    c = cases.four_quadrant(nx, seed=3, ny=ny)
    r = np.random.default_rng(seed)
    U = c.conserved() * (1.0 + 0.05 * r.standard_normal((4, ny, nx)))
    U[3] += 2.0  # keeps the pressure positive
    if nm == 1:
        return c, U
    d = 0.01 * r.standard_normal((4, nm, ny, nx))
    d[:, 0] = U
    return c, d


@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("spike", [False, True])
def test_weno_max_speed(restatement, ny, nx, spike):
    c, U = state(ny, nx, 1, 5)
    if spike:
        U[1, ny // 2, nx - 1] = 50.0
        U[3, ny // 2, nx - 1] = 5000.0
        U[0, 0, 0] = np.nan  # a NaN speed never wins
    with Solver(method="weno") as s:
        s.set_mesh(ny, nx, c.da, c.gamma, c.bctype)
        s.set_state(U)
        assert s.max_speed() == restatement.weno_max_speed(U, c.gamma)


@pytest.mark.parametrize("P", [1, 2, 3])
@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("inflow", [False, True])
def test_dg_max_speed(restatement, P, ny, nx, inflow):
    c, d = state(ny, nx, (P + 1) ** 2, 6)
    b = c.bctype.copy()
    if inflow:  # frozen bctype-0 cells outside the updated range count too
        b[3:-3, :3] = 0
        b[3:-3, -1] = 0
        d[1, 0, ny // 2, nx - 1] = 50.0
        d[3, 0, ny // 2, nx - 1] = 5000.0
    with Solver(method="dg", order=P) as s:
        s.set_mesh(ny, nx, c.da, c.gamma, b)
        s.set_state(d)
        assert s.max_speed() == restatement.dg_max_speed(P, d, b, c.gamma)

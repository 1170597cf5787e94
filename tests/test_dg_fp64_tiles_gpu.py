"""FP64 DG tiles at the edges: widths around the 32-cell row segments, the
smallest grid, slip walls on both sides of a segment boundary, states that
drive every branch of the limiter, a NaN cell.

The oracle performs the same operations in the same order, so everything made
of + - * / sqrt is compared for equality.  The reference limiter's filter uses
log10 and sin, whose last bit may differ between the two math libraries: those
runs are held to the 1e-12 of the golden tests.
"""
import numpy as np
import pytest

from conftest import rel_linf
from zuikakucfd_b200 import Solver, cases

pytestmark = pytest.mark.gpu

SIZES = [(7, 7), (9, 31), (10, 32), (8, 33), (12, 35), (9, 70)]


def problem(P, ny, nx, walls, seed, amp=0.02):
    c = cases.four_quadrant(nx, seed=4, ny=ny)
    r = np.random.default_rng(seed)
    d = amp * r.standard_normal((4, (P + 1) ** 2, ny, nx))
    d[:, 0] = c.conserved() * (1.0 + 0.02 * r.standard_normal((4, ny, nx)))
    b = c.bctype.copy()
    if walls:
        b[:3, :] = 1            # slip wall on top
        b[ny // 2, 3:5] = 1     # an obstacle at the left edge
        if nx > 40:
            b[ny // 2 - 1:ny // 2 + 1, 31:33] = 1  # and one across a segment boundary
    return c, d, b


def open_solver(P, c, b, **kw):
    s = Solver(method="dg", order=P, **kw)
    s.set_mesh(c.ny, c.nx, c.da, c.gamma, b)
    return s


@pytest.mark.parametrize("P", [1, 2, 3])
@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("walls,hll", [(False, False), (True, False), (True, True)])
def test_rhs_and_unlimited_step(restatement, P, ny, nx, walls, hll):
    c, d, b = problem(P, ny, nx, walls, 7)
    dt = 1e-3 * c.da
    with open_solver(P, c, b, limiter="none", flux="hll" if hll else "hllc") as s:
        s.set_state(d)
        s.step(dt, 2)
        out = s.get_state()
        s.set_state(d)
        dU = s.rhs(0.0)
    ref = restatement.dg_step_lim(P, d.copy(), b, c.da, c.gamma, dt, 2, limiter="none", hll=hll)
    assert np.isfinite(ref).all() and np.array_equal(out, ref)
    assert np.array_equal(dU, restatement.dg_rhs(P, d.copy(), b, c.da, c.gamma, hll=hll)[1])


@pytest.mark.parametrize("P", [1, 2, 3])
@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("amp", [1e-9, 0.02, 0.6])
def test_reference_limiter(restatement, P, ny, nx, amp):
    """amp 1e-9: nothing fires; 0.02: the modal filter; 0.6: both positivity
    passes, with negative densities and pressures at many points."""
    c, d, b = problem(P, ny, nx, False, 8, amp)
    if amp == 0.6:
        d[:3, 0, ny // 2, nx // 2] = 1e-7, 1e-4, 1e-4  # mean floors
        d[3, 0, ny // 2, 3] = 1e-3
    with open_solver(P, c, b) as s:
        s.set_state(d)
        s.limit()
        out = s.get_state()
    ref = restatement.dg_limit(P, d.copy(), b, c.gamma)
    assert rel_linf(out, ref) <= 1e-12


@pytest.mark.parametrize("P", [1, 3])
def test_nan_spreads_as_in_the_oracle(restatement, P):
    c, d, b = problem(P, 12, 70, False, 9)
    d[1, 1, 6, 32] = np.nan
    d[3, 0, 6, 40] = np.inf
    with open_solver(P, c, b, limiter="none") as s:
        s.set_state(d)
        s.step(1e-3 * c.da, 1)
        out, word = s.get_state(), s.status_word()
    ref = restatement.dg_step_lim(P, d.copy(), b, c.da, c.gamma, 1e-3 * c.da, 1, limiter="none")
    assert word & 1
    assert np.array_equal(np.isfinite(out), np.isfinite(ref))
    assert np.array_equal(out[np.isfinite(ref)], ref[np.isfinite(ref)])


@pytest.mark.parametrize("P", [1, 2, 3])
@pytest.mark.parametrize("kind", ["huge", "tiny", "rest"])
def test_operands_outside_the_branch_free_division(restatement, P, kind):
    """Values beyond the shared-reciprocal range next to ordinary ones, and a
    gas at rest (zero momenta): both divisions round alike."""
    c, d, b = problem(P, 12, 70, True, 10)
    r = np.random.default_rng(11)
    if kind == "huge":
        d[:, :, :, 35:] *= 2.0 ** 110
    elif kind == "tiny":
        d[1:3] = r.choice([0.0, -0.0, 5e-324, 1e-310, 1e-120, 1e-95, -1e-90, 1e-20], size=d[1:3].shape)
    else:
        d[1:3] = 0.0
        d[:, 1:] = 0.0
    dt = 1e-3 * c.da
    with open_solver(P, c, b, limiter="none") as s:
        s.set_state(d)
        s.step(dt, 1)
        out = s.get_state()
    ref = restatement.dg_step_lim(P, d.copy(), b, c.da, c.gamma, dt, 1, limiter="none")
    assert np.array_equal(out, ref, equal_nan=True)

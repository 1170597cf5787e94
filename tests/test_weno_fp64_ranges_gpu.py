"""FP64 WENO stages whose operands leave the branch-free division's range, and
tiles at their edges: bit-equal to the oracle.

The kernel divides by a shared reciprocal where operands are within fixed
powers of two and by plain division elsewhere; both round as IEEE division
does, so every case is compared for equality (infinities and NaN included).
"""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver, cases

pytestmark = pytest.mark.gpu

SIZES = [(7, 7), (8, 31), (9, 32), (17, 33), (16, 70)]


def perturbed(ny, nx, seed):
    c = cases.four_quadrant(nx, seed=2, ny=ny)
    r = np.random.default_rng(seed)
    return c, c.conserved() * (1.0 + 0.1 * r.standard_normal((4, ny, nx))), r


def magnitudes(kind, U, r):
    ny, nx = U.shape[1:]
    if kind == "plain":
        return U
    if kind == "huge":        # weights' squares and conserved values beyond the range
        U = U * 1.0
        U[:, :, nx // 2:] *= 2.0 ** 70
        U[:, ny // 2:, :] *= 2.0 ** 60
        return U
    if kind == "tiny":        # momenta 0, -0, denormal and below 2^-300 beside ordinary ones
        U[1:3] = r.choice([0.0, -0.0, 5e-324, 1e-310, 1e-120, 1e-90, -1e-91, 1e-20, 0.3], size=(2, ny, nx))
        U[3] += 1.0
        return U
    if kind == "vacuum":      # floored densities and pressures, supersonic faces, zero denominators
        U[0] = np.where(r.random((ny, nx)) < 0.3, 1e-14, U[0])
        U[1] *= 30.0
        return U
    U[2, ny // 2, nx // 2] = np.nan
    U[3, ny // 2, 3] = np.inf
    return U


# one ragged size per tile: 2 rows (the sizes above), 8 rows wide, 16 and 8
@pytest.mark.parametrize("ny,nx", SIZES + [(97, 201), (173, 301), (241, 517)])
@pytest.mark.parametrize("kind", ["plain", "huge", "tiny", "vacuum", "nonfinite"])
def test_weno_step_bits(restatement, ny, nx, kind):
    c, U, r = perturbed(ny, nx, 3)
    U = magnitudes(kind, U, r)
    dt = 1e-3 * c.da
    with np.errstate(all="ignore"):
        ref = restatement.weno_step(U.copy(), c.bctype, c.da, c.gamma, dt, 1)
    with Solver(method="weno") as s:
        s.set_mesh(ny, nx, c.da, c.gamma, c.bctype)
        s.set_state(U)
        s.step(dt, 1)
        out = s.get_state()
    assert np.array_equal(out, ref, equal_nan=True)


@pytest.mark.parametrize("recon", ["muscl_minmod", "muscl_vanleer", "muscl_superbee"])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_muscl_step_bits(restatement, ny, nx, recon):
    from zuikakucfd_b200 import _native as N
    c, U, _ = perturbed(ny, nx, 4)
    code = N.RECON[recon]
    ref = restatement.weno_step(U.copy(), c.bctype, c.da, c.gamma, 1e-3 * c.da, 2, recon=code)
    with Solver(method="weno", recon=recon) as s:
        s.set_mesh(ny, nx, c.da, c.gamma, c.bctype)
        s.set_state(U)
        s.step(1e-3 * c.da, 2)
        assert np.array_equal(s.get_state(), ref)

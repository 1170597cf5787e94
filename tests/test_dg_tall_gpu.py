"""FP64 and FP64_FMA DG on more rows than gridDim.y counts (65,535): the first
and the last rows of a tall grid come out as those of a short one."""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver

pytestmark = pytest.mark.gpu

NX, SHORT, KEEP = 9, 64, 50  # two steps reach 6 rows


def stepped(U, precision, limiter):
    ny = U.shape[2]
    b = np.full((ny, NX), -1, np.int32)
    b[3:-3, 3:-3] = 0
    with Solver(method="dg", order=1, precision=precision, limiter=limiter) as s:
        s.set_mesh(ny, NX, 1.0 / NX, 1.4, b)
        s.set_state(U)
        s.step(1e-3, 2)
        return s.get_state()


@pytest.mark.parametrize("precision", ["fp64", "fp64_fma"])
@pytest.mark.parametrize("limiter", ["reference", "none"])
@pytest.mark.parametrize("ny", [65_536, 65_541])  # one row more in the cell pass, in both
def test_tall_grid(precision, limiter, ny):
    r = np.random.default_rng(3)
    U = 0.02 * r.standard_normal((4, 4, ny, NX))
    U[:, 0] += np.array([1.0, 0.3, 0.2, 2.5])[:, None, None]
    out = stepped(U, precision, limiter)
    assert np.isfinite(out).all()
    assert np.array_equal(out[:, :, :KEEP], stepped(U[:, :, :SHORT].copy(), precision, limiter)[:, :, :KEEP])
    assert np.array_equal(out[:, :, -KEEP:], stepped(U[:, :, -SHORT:].copy(), precision, limiter)[:, :, -KEEP:])

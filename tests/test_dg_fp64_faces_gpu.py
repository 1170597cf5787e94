"""The FP64 DG face pass with one Gauss point per thread (few CTAs) and with
several, on both sides of the line between them on 148 SMs (296 CTAs)."""
import numpy as np
import pytest

from test_dg_fp64_tiles_gpu import open_solver, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 2, 3])
@pytest.mark.parametrize("ny,nx", [(103, 70), (104, 70), (301, 31), (302, 31)])  # 294, 297, 296, 297 CTAs
@pytest.mark.parametrize("walls,hll", [(False, False), (True, True)])
def test_both_splits_of_the_points(restatement, P, ny, nx, walls, hll):
    c, d, b = problem(P, ny, nx, walls, 12)
    dt = 1e-3 * c.da
    kw = dict(limiter="none", flux="hll" if hll else "hllc")
    with open_solver(P, c, b, **kw) as s:
        s.set_state(d)
        s.step(dt, 1)
        out = s.get_state()
    ref = restatement.dg_step_lim(P, d.copy(), b, c.da, c.gamma, dt, 1, limiter="none", hll=hll)
    assert np.isfinite(ref).all() and np.array_equal(out, ref)
    with open_solver(P, c, b, precision="fp64_fma", **kw) as s:
        s.set_state(d)
        s.step(dt, 1)
        assert np.abs(s.get_state() - ref).max() <= 1e-12 * np.abs(ref).max()

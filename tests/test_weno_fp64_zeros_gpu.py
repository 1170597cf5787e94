"""FP64 WENO and MUSCL steps on states with momenta of either zero: the
oracle's bits, the signs of zeros included."""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver, _native as N, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recon", ["weno5", "muscl_minmod", "muscl_vanleer", "muscl_superbee"])
@pytest.mark.parametrize("ny,nx", [(7, 7), (17, 33), (97, 201)])
@pytest.mark.parametrize("share", [0.5, 1.0])  # of the momenta that are zeros
def test_step_bits(restatement, ny, nx, recon, share):
    c = cases.four_quadrant(nx, seed=2, ny=ny)
    r = np.random.default_rng(7)
    U = c.conserved() * (1.0 + 0.1 * r.standard_normal((4, ny, nx)))
    zeros = r.choice([0.0, -0.0], size=(2, ny, nx))
    U[1:3] = np.where(r.random((2, ny, nx)) < share, zeros, U[1:3])
    ref = restatement.weno_step(U.copy(), c.bctype, c.da, c.gamma, 1e-3 * c.da, 2, recon=N.RECON[recon])
    with Solver(method="weno", recon=recon) as s:
        s.set_mesh(ny, nx, c.da, c.gamma, c.bctype)
        s.set_state(U)
        s.step(1e-3 * c.da, 2)
        out = s.get_state()
    assert np.isfinite(ref).all()
    assert np.array_equal(out.view(np.uint64), ref.view(np.uint64))

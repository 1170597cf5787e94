"""A launch the grid limits refuse is reported once: the context's next call
runs as if it had not been tried."""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver
from zuikakucfd_b200._native import ZkError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_calls_after_a_refused_launch(precision):
    ny, nx = 8 * 65535 + 1, 7  # one 8-row tile more than gridDim.y counts
    b = np.full((ny, nx), -1, np.int32)
    b[3:-3, 3:-3] = 0
    U = np.empty((4, ny, nx))
    U[:] = np.array([1.0, 0.3, 0.2, 2.5])[:, None, None]
    with Solver(method="weno", precision=precision) as s:
        s.set_mesh(ny, nx, 1.0 / nx, 1.4, b)
        s.set_state(U)
        lam = s.max_speed()
        with pytest.raises(ZkError, match="invalid"):
            s.step(1e-3, 1)
        assert s.max_speed() == lam
        assert np.array_equal(s.recover_primitives()[0], U[0])

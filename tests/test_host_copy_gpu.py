"""State copies large enough to be staged by host threads: what goes in comes
out, at widths that leave ragged chunks and with the padding columns of the
device rows untouched, from pageable and page-locked arrays."""
import numpy as np
import pytest

from zuikakucfd_b200 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,ny,nx", [(3, 301, 299), (3, 7, 20_011), (2, 1000, 97), (1, 2100, 1030)])
def test_state_round_trip(order, ny, nx):
    import torch
    r = np.random.default_rng(order)
    b = np.zeros((ny, nx), np.int32)
    with Solver(method="dg", order=order) as s:
        s.set_mesh(ny, nx, 1.0 / nx, 1.4, b)
        for k in range(3):  # the first read allocates the staging; later copies both use it
            U = r.random(s.state_shape)
            if k == 2:
                U = torch.from_numpy(U).pin_memory().numpy()
            s.set_state(U)
            assert np.array_equal(s.get_state(), U)
        s.set_state(U)
        prim = s.recover_primitives()
        assert np.array_equal(prim[0], U[0, 0])

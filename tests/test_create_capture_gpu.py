"""zk_create while another stream is being captured: it succeeds and leaves the
capture sound (a context allocates memory with its mesh, not before)."""
import pytest

from zuikakucfd_b200 import Solver

pytestmark = pytest.mark.gpu


def test_create_during_a_capture():
    import torch
    x = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x += 1.0
        s = Solver(method="weno")
    g.replay()
    torch.cuda.synchronize()
    assert (x == 1.0).all()
    s.close()

"""Large host copies on streams other than the context's own.  A stream handle
can mean different streams in different threads (cudaStreamPerThread), and
another stream may be being captured while the copy runs."""
import threading

import numpy as np
import pytest

from zuikakucfd_b200 import Solver, cases

pytestmark = pytest.mark.gpu

LEGACY, PER_THREAD = 1, 2  # cudaStreamLegacy, cudaStreamPerThread
NY, NX = 1200, 1001        # DG P=1: 154 MB, recovered primitives 38 MB


def problem(seed):
    c = cases.four_quadrant(NX, seed=2, ny=NY)
    r = np.random.default_rng(seed)
    d = 0.01 * r.standard_normal((4, 4, NY, NX))
    d[:, 0] = c.conserved() * (1.0 + 0.02 * r.standard_normal((4, NY, NX)))
    return c, d


def opened(c):
    s = Solver(method="dg", order=1, limiter="none")
    s.set_mesh(c.ny, c.nx, c.da, c.gamma, c.bctype)
    return s


def calls(s, d):
    """Every call that ends in a staged copy, right behind the kernel it reads from."""
    s.set_state(d)
    out = [s.get_state(), s.recover_primitives(), s.rhs(0.0)]  # rhs fills the ghosts
    s.set_state(2.0 * d)  # staged from here on
    s.set_state(d)
    return out + [s.get_state(), s.rhs(0.0)]


@pytest.mark.parametrize("handle", [LEGACY, PER_THREAD])
def test_shared_handles(handle):
    c, d = problem(1)
    with opened(c) as s:
        ref = calls(s, d)
    got = {}
    with opened(c) as s:
        s.set_stream(handle)

        def take(k):
            got[k] = [calls(s, d) for _ in range(2)]

        for k in range(2):  # from two host threads in turn
            t = threading.Thread(target=take, args=(k,))
            t.start()
            t.join()
    for k in range(2):
        for run in got[k]:
            for a, b in zip(run, ref):
                assert np.array_equal(a, b)


def test_first_copy_during_another_streams_capture():
    """The first large copy page-locks its buffers, which may not disturb a
    capture under way on another stream."""
    import torch
    c, _ = problem(2)
    with opened(c) as s:
        x = torch.zeros(1024, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="global"):
            x += 1.0
            out = s.get_state()
        g.replay()
        torch.cuda.synchronize()
        assert (x == 1.0).all() and not out.any()

"""A device reset elsewhere in the process: what was uploaded or set for the old
CUDA context is set up again for contexts created afterwards.

In a process of its own, since the reset takes every other allocation with it."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes
import numpy as np
from zuikakucfd_b200 import Solver, cases
from zuikakucfd_b200.batch import Batch

c = cases.four_quadrant(70, seed=3, ny=41)

def state(order):
    U = np.zeros((4, (order + 1) ** 2, c.ny, c.nx))
    U[:, 0] = c.conserved()
    return U if order else U[:, 0]

def results():
    out = []
    for method, order, precision, tpc in [("weno", 0, "fp64", 0), ("weno", 0, "fp64_fma", 0), ("weno", 0, "mixed", 0),
                                          ("dg", 1, "fp64", 0), ("dg", 2, "fp64_fma", 0), ("dg", 3, "fp64", 0),
                                          ("dg", 1, "mixed", 1), ("dg", 2, "mixed", 2), ("dg", 3, "mixed", 1),
                                          ("dg", 3, "mixed", 2)]:
        with Solver(method=method, order=max(order, 1), precision=precision, tile_tpc=tpc) as s:
            s.set_mesh(c.ny, c.nx, c.da, c.gamma, c.bctype)
            s.set_state(state(order))
            s.step(1e-3 * c.da, 2)
            out.append(s.get_state())
    with Batch(policy="all", autotune=0) as b:
        ids = [b.add(c.bctype, c.da, c.gamma, state(2 if m == "dg" else 0), 2, 0.4, method=m, order=2, precision=p)
               for m in ("weno", "dg") for p in ("fp64", "mixed")]
        b.run()
        out += [b.get_state(k) for k in ids]
    return out

before = results()
assert ctypes.CDLL(RESET).reset() == 0
after = results()
assert len(before) == len(after) == 14
for k, (x, y) in enumerate(zip(before, after)):
    assert np.isfinite(x).all() and np.array_equal(x, y), k
print("ok")
"""


def test_contexts_after_a_device_reset(tmp_path):
    from zuikakucfd_b200 import build
    # the primary context is reset through a runtime of the test's own
    src, so = tmp_path / "reset.cu", tmp_path / "reset.so"
    src.write_text('#include <cuda_runtime.h>\nextern "C" int reset() { return cudaDeviceReset(); }\n')
    subprocess.run([build.nvcc(), "-shared", "-Xcompiler", "-fPIC", "-cudart", "static", "-o", str(so), str(src)],
                   check=True, capture_output=True)
    script = f"RESET = {str(so)!r}\n" + SCRIPT
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]

"""The branch-free FP64 division against plain division, bit for bit, and the
bound on the hardware reciprocal that its proof starts from."""
import ctypes
import subprocess

import numpy as np
import pytest

from zuikakucfd_b200 import build

pytestmark = pytest.mark.gpu

ONES = (1 << 52) - 1
N = 1 << 20


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("div") / "check.so"
    src = build.ROOT / "tests" / "fp64_div_check.cu"
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, *build.STRICT, "-shared", "-cudart", "static",
                    "-o", str(so), str(src)], check=True, capture_output=True)
    fn = ctypes.CDLL(str(so)).fp64_div_check
    D = ctypes.POINTER(ctypes.c_double)
    fn.argtypes = [ctypes.c_int, D, D, D]

    def call(a, b):
        a, b = np.ascontiguousarray(a, float), np.ascontiguousarray(b, float)
        out = np.empty((9, a.size))
        assert fn(a.size, *(x.ctypes.data_as(D) for x in (a, b, out))) == 0
        return dict(zip(["seed", "recip", "quot", "divide", "one_over", "plain", "residual", "in_range", "num_ok"],
                        out))

    return call


def compose(sig, exp, sign=0):
    bits = (np.asarray(exp, np.int64) + 1023 << 52) | np.asarray(sig, np.int64) | (np.asarray(sign, np.int64) << 63)
    return np.broadcast_to(bits, (N,)).copy().view(np.float64)


def significands(kind, r):
    """[0, 2^52) with, by kind, the shapes where a last bit goes wrong."""
    any_ = r.integers(0, 1 << 52, N)
    if kind == "ones":          # the neighbours of the all-ones significand, itself among them
        return ONES - r.integers(0, 1 << 12, N)
    if kind == "power":         # just above a power of two
        return r.integers(0, 1 << 12, N)
    if kind == "short":         # few significant bits: exact quotients and ties
        return any_ >> 40 << 40
    if kind == "hole":          # all ones but one bit
        return ONES ^ (1 << r.integers(0, 52, N))
    return any_


@pytest.mark.parametrize("exp", [-500, -41, 0, 1, 333, 499])
def test_seed(check, exp):
    """|1 - b seed| < 2^-19 for all 2^20 leading parts of a significand, at
    both ends of the remaining 32 bits and inside."""
    r = np.random.default_rng(exp + 500)
    hi = np.arange(N) << 32
    for lo in (0, 0xffffffff, r.integers(0, 1 << 32, N)):
        got = check(np.ones(N), compose(hi + lo, exp))
        assert np.abs(got["residual"]).max() < 2.0 ** -19


@pytest.mark.parametrize("kind_a", ["any", "ones", "power", "short", "near_b"])
@pytest.mark.parametrize("kind_b", ["any", "ones", "power", "short", "hole"])
# exponents of a and b: one binade; the bounds of num_ok and in_range; a state's
# own quotients' quotients by a density or a wave-speed difference
@pytest.mark.parametrize("ea,eb", [((0, 1), (0, 1)), ((-300, 100), (-500, 500)), ((-720, 400), (-60, 220))])
def test_quotients_are_those_of_plain_division(check, kind_a, kind_b, ea, eb):
    r = np.random.default_rng([ord(kind_a[0]), ord(kind_b[0]), ea[0] + 1000])
    sb = significands(kind_b, r)
    sa = np.clip(sb + r.integers(-8, 9, N), 0, ONES) if kind_a == "near_b" else significands(kind_a, r)
    a = compose(sa, r.integers(*ea, N), r.integers(0, 2, N))
    b = compose(sb, r.integers(*eb, N), r.integers(0, 2, N))
    got = check(a, b)
    ok = (sb & 0xffffffff) != 0xffffffff
    assert np.array_equal(got["in_range"] == 1, ok)
    if ea == (-300, 100):
        assert (got["num_ok"] == 1).all()
    bits = {k: v.view(np.uint64)[ok] for k, v in got.items()}
    assert np.array_equal(bits["recip"], bits["one_over"])
    assert np.array_equal(bits["divide"], bits["plain"])
    pos = (b > 0)[ok]
    assert np.array_equal(bits["quot"][pos], bits["plain"][pos])


def test_signed_zeros(check):
    """quot keeps the sign of either zero over a positive denominator, divide
    that of +0 over any."""
    r = np.random.default_rng(1)
    b = compose(significands("any", r), r.integers(-60, 220, N), r.integers(0, 2, N))
    a = np.where(r.integers(0, 2, N) == 1, 0.0, -0.0)
    ok = (b.view(np.uint64) & 0xffffffff) != 0xffffffff
    for name, sel in (("quot", ok & (b > 0)), ("divide", ok & ~np.signbit(a))):
        got = check(a[sel], b[sel])
        assert np.array_equal(got[name].view(np.uint64), got["plain"].view(np.uint64)), name

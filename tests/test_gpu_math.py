"""The scalar helpers of the step kernels (wdem_math.cuh) on every exponent, with zeros, subnormals, infinities and NaN.

Reciprocal and roots: one step of third order from a seed within 2^-21.9 leaves a truncation error below 2^-65 and
roundings of terms below 2^-21 of the result, so the result is within 0.5 ulp and 2^-12 of one; the square root's last
step doubles its digits.  Held to 0.501 ulp of the exact value in extended precision (64 or 113 bits).  Outside exponents
4 to 2040, and for arguments without a root, they are CUDA's operations, bit for bit.  The bit tricks equal the FP64
operations they stand for, bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from woo_gb300 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
RECIP, RSQRT, SQRT, HALF, TWICE, PLUS_ZERO, FLIP, GREATER, BELOW, PICK, CUDA_RECIP, CUDA_RSQRT, CUDA_SQRT = range(13)


@pytest.fixture(scope="module")
def math_lib(wdem_lib, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("math") / "libmath.so")
    flags = [f for f in build.FLAGS if f != "--fmad=false"]
    subprocess.run([build.nvcc(), *build.ARCH, *flags, "-DWDEM_FMA", "--fmad=true", "-shared",
                    os.path.join(HERE, "native", "math_check.cu"), "-o", out, "-lcudart"], check=True)
    return ctypes.CDLL(out)


P = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def evaluate(math_lib):
    def run(what, x, y=None):
        x = np.ascontiguousarray(x)
        y = x if y is None else np.ascontiguousarray(y)
        r = np.empty(len(x))
        assert math_lib.math_eval(what, x.ctypes.data_as(P), y.ctypes.data_as(P), r.ctypes.data_as(P), len(x)) == 0
        return r
    return run


def _arguments(per=64):
    """Every exponent with random and extreme significands, both signs; zeros, infinities, NaN."""
    rng = np.random.default_rng(1)
    e = np.repeat(np.arange(2048, dtype=np.uint64), per)
    m = rng.integers(0, 1 << 52, len(e), dtype=np.uint64)
    m[0::per], m[1::per], m[2::per], m[3::per] = 0, 1, (1 << 52) - 1, 1 << 51
    sign = rng.integers(0, 2, len(e), dtype=np.uint64)
    sign[0::2 * per] = 0
    return ((sign << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


def _same(a, b):
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


def _exponent(x):
    return ((x.view(np.uint64) >> np.uint64(52)) & np.uint64(2047)).astype(int)


@pytest.mark.parametrize("fast, cuda", [(RECIP, CUDA_RECIP), (RSQRT, CUDA_RSQRT), (SQRT, CUDA_SQRT)])
def test_reciprocal_and_roots(evaluate, fast, cuda):
    x = _arguments()
    r = evaluate(fast, x)
    e = _exponent(x)
    inside = (e >= 4) & (e <= 2040) & ((x > 0) | (fast == RECIP))
    assert _same(r, evaluate(cuda, x))[~inside].all()
    # many more arguments in the range the contact law meets
    rng = np.random.default_rng(2)
    more = np.ldexp(rng.uniform(1, 2, 1 << 20), rng.integers(-60, 60, 1 << 20))
    for a in (x[inside], more):
        v = evaluate(fast, a)
        L = a.astype(np.longdouble)
        exact = 1 / L if fast == RECIP else (1 / np.sqrt(L) if fast == RSQRT else np.sqrt(L))
        ulp = np.ldexp(1.0, np.frexp(np.abs(exact).astype(np.float64))[1] - 53)
        normal = np.abs(v) >= 2.0 ** -1022
        assert normal.all()
        assert (np.abs(v - exact) / ulp).max() <= 0.501


def test_bit_tricks(evaluate):
    x = _arguments(16)
    rng = np.random.default_rng(3)
    y = rng.permutation(x)
    y[::3] = x[::3]
    with np.errstate(all="ignore"):
        y[1::9] = np.nextafter(x[1::9], np.inf)
        assert _same(evaluate(HALF, x), 0.5 * x).all()
        assert _same(evaluate(TWICE, x), x + x).all()
        assert _same(evaluate(PLUS_ZERO, x), x + 0.0).all()
        assert _same(evaluate(FLIP, x), -x).all()
        number = ~np.isnan(x) & ~np.isnan(y)
        assert np.array_equal(evaluate(GREATER, x, y)[number], (x > y)[number].astype(float))
        hi = (np.abs(x).view(np.uint64) >> np.uint64(32))
        bound = np.array([1e-8]).view(np.uint64)[0] >> np.uint64(32)
        assert np.array_equal(evaluate(BELOW, x), (hi < bound).astype(float))
        odd = np.arange(len(x)) & 1
        assert _same(evaluate(PICK, x, y), np.where(odd, x, y)).all()


def _quaternion(c):
    """Shoemake's four cases of the frames with columns c[:, 0], c[:, 1], c[:, 2], in c's precision; the case taken as
    FP64 sees it."""
    m = [[c[:, k, r] for k in range(3)] for r in range(3)]
    f = [m[k][k].astype(np.float64) for k in range(3)]
    pos = f[0] + f[1] + f[2] > 0
    big = np.argmax(np.stack(f), axis=0)
    case = np.where(pos, 3, big)
    one = c.dtype.type(1)
    q = np.empty((len(c), 4), c.dtype)  # w, x, y, z
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        s = case == i
        t = np.sqrt(m[i][i] - m[j][j] - m[k][k] + one)
        h = one / 2 / t
        q[s, 1 + i] = (t / 2)[s]
        q[s, 0] = ((m[k][j] - m[j][k]) * h)[s]
        q[s, 1 + j] = ((m[j][i] + m[i][j]) * h)[s]
        q[s, 1 + k] = ((m[k][i] + m[i][k]) * h)[s]
    t = np.sqrt(np.where(pos, m[0][0] + m[1][1] + m[2][2], 0) + one)
    h = one / 2 / t
    q[pos, 0] = (t / 2)[pos]
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        q[pos, 1 + i] = ((m[k][j] - m[j][k]) * h)[pos]
    return q


def test_quaternion_of_a_frame(math_lib):
    """The contact frame's quaternion carries no larger root mean square error than the same formulas with IEEE square
    root and division."""
    rng = np.random.default_rng(5)
    n = 1 << 18
    a, b = rng.normal(size=(2, n, 3)).astype(np.longdouble)
    a /= np.sqrt((a * a).sum(1, keepdims=True))
    b -= (a * b).sum(1, keepdims=True) * a
    b /= np.sqrt((b * b).sum(1, keepdims=True))
    c = np.ascontiguousarray(np.stack([a, b, np.cross(a, b)], axis=1).astype(np.float64))
    got = np.empty((n, 4))
    assert math_lib.quat_eval(c.ctypes.data_as(P), got.ctypes.data_as(P), n) == 0
    with np.errstate(invalid="ignore", divide="ignore"):
        exact, ieee = _quaternion(c.astype(np.longdouble)), _quaternion(c)
    rms = [float(np.sqrt(((q - exact) ** 2).sum(1).mean())) for q in (got, ieee)]
    assert np.abs(got - exact).max() < 1e-15
    assert rms[0] <= rms[1], rms

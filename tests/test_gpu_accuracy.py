"""Rounding error of the mixed-radix lines against extended precision, line
lengths whose radices are odd above all. Each case states the rel-L2 error that
the kernels before the mixed-radix tiles (one prime radix a stage, one table
product a four-step output) had on B200 for U[-1, 1) lines; the tiles
may not be less exact. Bound: that figure plus 2%, of which sampling takes
about 1% (the figures come from 60000 points, the test takes at least 120000: the
relative spread of a root mean square over P independent errors is below
1 / sqrt(P) = 0.3%, three of them)."""
import ctypes as C

import numpy as np
import pytest
import scipy.fft

import aoclfftz_b200
from aoclfftz_b200 import synthetic
from fftz_helpers import cplx_dtype, run_gpu

pytestmark = pytest.mark.gpu


def exact(x, kind, n, direction):
    """The transform of each row in long double (of a float line in double)."""
    x = x.astype({"f": np.float64, "d": np.longdouble, "F": np.complex128, "D": np.clongdouble}[x.dtype.char])
    if kind == "c2c":
        return scipy.fft.fft(x) if direction == 0 else scipy.fft.ifft(x, norm="forward")
    return scipy.fft.rfft(x) if direction == 0 else scipy.fft.irfft(x, n=n, norm="forward")


def rel_error(kind, dtype, n, direction, lines):
    half = n // 2 + 1
    if kind == "c2c":
        x = synthetic.complex_uniform(n, n * lines, cplx_dtype(dtype)).reshape(lines, n)
        y, _ = run_gpu(dtype, [(n, 1, 1)], [(lines, n, n)], x, 2 * n * lines, 0, direction)
        y = y.view(cplx_dtype(dtype)).reshape(lines, n)
    else:
        x = synthetic.complex_uniform(n, half * lines, cplx_dtype(dtype)).reshape(lines, half)
        if direction == 0:
            x = np.ascontiguousarray(x.view(x.real.dtype)[:, :n])
            y, _ = run_gpu(dtype, [(n, 1, 1)], [(lines, n, half)], x, 2 * half * lines, 1, 0)
            y = y.view(cplx_dtype(dtype)).reshape(lines, half)
        else:
            x[:, 0] = x[:, 0].real
            if n % 2 == 0:
                x[:, -1] = x[:, -1].real
            y, _ = run_gpu(dtype, [(n, 1, 1)], [(lines, half, n)], x, n * lines, 1, 1)
            y = y.reshape(lines, n)
    ref = exact(x, kind, n, direction)
    return float(np.sqrt((np.abs(y - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()))


def check(kind, dtype, n, direction, former):
    err = rel_error(kind, dtype, n, direction, max(1, -(-120000 // n)))
    assert err <= 1.02 * former, "rel-L2 %.3e, formerly %.3e (%.3f)" % (err, former, err / former)


@pytest.mark.parametrize("kind,dtype,n,direction,former", [
    ("c2c", "f32", 81, 0, 9.31e-8), ("c2c", "f32", 729, 1, 1.194e-7), ("c2c", "f32", 2187, 1, 1.302e-7),
    ("c2c", "f32", 6561, 1, 1.417e-7), ("c2c", "f64", 2187, 1, 2.765e-16), ("real", "f32", 2187, 1, 1.054e-7),
    ("real", "f32", 6561, 0, 1.396e-7), ("real", "f32", 6561, 1, 1.124e-7), ("real", "f64", 2187, 0, 2.641e-16),
    ("real", "f64", 8192, 0, 2.425e-16), ("real", "f64", 8192, 1, 2.415e-16)])
def test_one_pass_lines(kind, dtype, n, direction, former):
    check(kind, dtype, n, direction, former)


@pytest.mark.parametrize("kind,dtype,n,direction,former", [
    ("c2c", "f32", 117649, 1, 1.600e-7), ("c2c", "f32", 177147, 1, 1.765e-7), ("c2c", "f32", 500000, 1, 1.652e-7),
    ("c2c", "f32", 531441, 1, 1.852e-7), ("c2c", "f64", 117649, 1, 2.879e-16), ("c2c", "f64", 161051, 1, 3.019e-16),
    ("c2c", "f64", 390625, 1, 3.163e-16), ("c2c", "f64", 531441, 1, 4.000e-16), ("real", "f64", 16807, 1, 2.008e-16)])
def test_four_step_lines(kind, dtype, n, direction, former):
    check(kind, dtype, n, direction, former)


@pytest.mark.parametrize("dtype,n,former", [
    ("f32", 17, 1.094e-7), ("f32", 101, 1.402e-7), ("f32", 521, 1.411e-7), ("f32", 1031, 1.528e-7),
    ("f32", 2053, 1.501e-7), ("f32", 3001, 1.701e-7), ("f32", 4099, 1.586e-7), ("f32", 5003, 1.683e-7),
    ("f32", 8209, 1.781e-7), ("f32", 10007, 1.860e-7), ("f32", 16411, 1.871e-7), ("f32", 20011, 1.951e-7),
    ("f32", 32771, 1.900e-7), ("f32", 262147, 2.020e-7), ("f64", 17, 2.113e-16), ("f64", 101, 3.025e-16),
    ("f64", 521, 3.243e-16), ("f64", 1031, 3.345e-16), ("f64", 2053, 3.772e-16), ("f64", 3001, 4.179e-16),
    ("f64", 4099, 3.991e-16), ("f64", 5003, 4.192e-16), ("f64", 8209, 4.032e-16), ("f64", 10007, 4.251e-16),
    ("f64", 16411, 4.057e-16), ("f64", 20011, 4.281e-16), ("f64", 32771, 4.438e-16), ("f64", 262147, 4.932e-16)])
def test_chirp_lengths(dtype, n, former):
    """Primes, most of them just above a power of two, whose convolution over the next power of two was the most exact
    (its noise spreads over twice the points); formerly: that power of two."""
    check("c2c", dtype, n, 1, former)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n", [3, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16])
def test_mean_gain_of_the_butterflies(n, dtype):
    """The gains that the stage tables take back (fz_mr_gain) are those of the butterflies: a column of n points is one.
    The mean over P outputs is exact to the error of one, a few times 2^-24 or 2^-53, over sqrt(P)."""
    lib = aoclfftz_b200.load()
    lib.fz_mr_gain.restype = C.c_double
    lines = 200000
    x = synthetic.complex_uniform(n, n * lines, cplx_dtype(dtype)).reshape(n, lines)
    y, _ = run_gpu(dtype, [(n, lines, lines)], [(lines, 1, 1)], x, 2 * n * lines)
    ref = exact(np.ascontiguousarray(x.T), "c2c", n, 0).T
    y = y.view(cplx_dtype(dtype)).reshape(n, lines)
    gain = float(((y - ref) * np.conj(ref)).real.sum() / (np.abs(ref) ** 2).sum())
    eps = 2.0 ** -24 if dtype == "f32" else 2.0 ** -53
    assert abs(gain - lib.fz_mr_gain(0 if dtype == "f32" else 1, n)) <= 8 * eps / np.sqrt(lines * n)

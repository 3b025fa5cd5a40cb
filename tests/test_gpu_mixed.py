"""GPU parity of the mixed-radix line kernel (csrc/kernels/fft_mr.cuh) against the
FP64 oracle at the edges of its shapes: one, two and more stages, every
composite radix, a last CTA that is not full, the longest line of each dtype,
row and column lane maps, non-unit strides, in place, four-step passes, real lines
with mirrored butterflies (odd and even butterfly counts, one stage, 11 and 13
alone) and unpacked odd ones.
Bound: rel-L2 <= 4 log2(n) eps of the working dtype (oracle.tol)."""
import pytest

from test_gpu_c2c import check_c2c
from test_gpu_real import check_real

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n,b", [(4, 5), (6, 700), (8, 1001), (9, 1), (10, 300), (16, 4097), (32, 77), (64, 3), (13, 33), (14, 129), (15, 7), (18, 65), (26, 50), (60, 301), (100, 41),
                                 (143, 9), (360, 14), (1000, 11), (1080, 3), (2187, 5), (11011, 2), (14400, 2)])
def test_rows(n, b, dtype):
    check_c2c(dtype, [(n, 1, 1)], [(b, n, n)], direction=n & 1, seed=n, compare_ref=False)


@pytest.mark.parametrize("dtype,n", [("f32", 28000), ("f32", 28800), ("f64", 14406)])
def test_longest_lines(dtype, n):
    check_c2c(dtype, [(n, 1, 1)], [(2, n, n)], seed=n, compare_ref=False)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n,b,place", [(12, 33, 1), (45, 5, 0), (375, 9, 1), (1080, 17, 0)])
def test_columns(n, b, place, dtype):
    check_c2c(dtype, [(n, b, b)], [(b, 1, 1)], direction=place, placement=place, seed=b, compare_ref=False)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_strides_and_mixed_maps(dtype):
    # rows in, columns out; then every second element in, every third out
    check_c2c(dtype, [(90, 1, 21)], [(21, 90, 1)], seed=3, compare_ref=False)
    check_c2c(dtype, [(70, 2, 3)], [(5, 150, 221)], seed=4, compare_ref=False)


@pytest.mark.parametrize("dtype,n,b", [("f32", 250047, 2), ("f64", 120000, 1), ("f32", 30030, 3)])
def test_four_step(dtype, n, b):
    check_c2c(dtype, [(n, 1, 1)], [(b, n, n)], direction=b & 1, seed=5, compare_ref=False)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("shape,batch", [((2,), 5), ((3,), 300), ((6,), 70), ((13,), 9), ((32,), 131), ((36,), 3), ((50,), 40),
                                         ((98,), 7), ((242,), 5), ((286,), 3), ((338,), 2), ((441,), 9), ((480,), 33),
                                         ((2048,), 5), ((14406,), 2), ((6, 9, 10), 2), ((17, 24), 3)])
def test_real_lines(shape, batch, dtype):
    check_real(dtype, shape, batch=batch, compare_ref=False)
    check_real(dtype, shape, batch=1, inplace=len(shape) > 1, compare_ref=False)


def test_longest_real_lines():
    check_real("f32", (56000,), batch=2, compare_ref=False)
    check_real("f64", (28800,), batch=1, compare_ref=False)

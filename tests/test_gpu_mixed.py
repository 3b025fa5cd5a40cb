"""GPU parity of the mixed-radix line kernel (csrc/kernels/fft_mr.cuh) against the
FP64 oracle at the edges of its shapes: one, two and more stages, every
composite radix, a last CTA that is not full, the longest line of each dtype,
row and column lane maps, non-unit strides, in place, four-step passes, real lines
with mirrored butterflies (odd and even butterfly counts, one stage, 11 and 13
alone, aligned and not) and unpacked odd ones, chirp-z on either side of the
one-kernel limit and in every layout, the older in-place kernel (kernel_family 12),
and launches captured into a graph.
Bound: rel-L2 <= 4 log2(n) eps of the working dtype (oracle.tol)."""
import ctypes as C

import numpy as np
import pytest

import aoclfftz_b200
import oracle
from aoclfftz_b200 import abi, synthetic
from fftz_helpers import cplx_dtype, real_dtype, run_gpu
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


@pytest.mark.parametrize("dtype,n,one", [("f32", 14401, True), ("f32", 14407, False), ("f64", 7193, True), ("f64", 7207, False)])
def test_chirp_at_the_one_kernel_limit(dtype, n, one):
    """2n - 1 is 28801 / 28813 and 14385 / 14413: the longest convolutions that fit a CTA are 28812 and 14406 points."""
    for direction in (0, 1):
        _, plan = check_c2c(dtype, [(n, 1, 1)], [(2, n, n)], direction=direction, seed=n, compare_ref=False)
        assert ("bluestein-mid" not in plan) == one, plan


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n,b", [(17, 70), (101, 21), (1009, 9), (14407, 3)])
def test_chirp_layouts(n, b, dtype):
    check_c2c(dtype, [(n, b, b)], [(b, 1, 1)], direction=n & 1, seed=n, compare_ref=False)               # columns
    check_c2c(dtype, [(n, 1, 1)], [(b, n + 3, n + 3)], placement=0, seed=n + 1, compare_ref=False)       # in place
    check_c2c(dtype, [(n, 2, 3)], [(b, 2 * n + 1, 3 * n + 5)], direction=1, seed=n + 2, compare_ref=False)  # strided
    check_c2c(dtype, [(n, 1, b)], [(b, n, 1)], seed=n + 3, compare_ref=False)                            # rows to columns


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n", [6, 32, 50, 98, 480])
def test_real_lines_off_the_pair_alignment(n, dtype):
    """Real rows an odd distance apart: every second one starts between two of the pairs that aligned rows move at once."""
    b, half, d = 7, n // 2 + 1, n + 1
    x = synthetic.normal(n, b * d).astype(real_dtype(dtype))
    raw, _ = run_gpu(dtype, [(n, 1, 1)], [(b, d, half)], x, 2 * b * half, 1, 0)
    X = raw.view(cplx_dtype(dtype)).reshape(b, half)
    rows = x.reshape(b, d)[:, :n].astype(np.float64)
    ref = oracle.rfftn(rows, rank=1)
    assert oracle.rel_l2(X, ref) <= oracle.tol(n, dtype)
    back, _ = run_gpu(dtype, [(n, 1, 1)], [(b, half, d)], ref.astype(cplx_dtype(dtype)), b * d, 1, 1)
    assert oracle.rel_l2(back.reshape(b, d)[:, :n], rows * n) <= oracle.tol(n, dtype)
    assert not back.reshape(b, d)[:, n].any()  # the gaps between the rows are not written


@pytest.fixture
def in_place_kernel():
    lib = aoclfftz_b200.load()
    h = abi.Hints()
    h.kernel_family = 12
    lib.aoclfftz_gpu_set_hints(C.byref(h))
    yield
    lib.aoclfftz_gpu_set_hints(None)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_in_place_kernel(dtype, in_place_kernel):
    for n, b in ((3, 9), (77, 5), (360, 14), (1080, 3), (2187, 2)):
        _, plan = check_c2c(dtype, [(n, 1, 1)], [(b, n, n)], direction=n & 1, seed=n, compare_ref=False)
        assert "[generic n=" in plan, plan
    check_c2c(dtype, [(100, 9, 9)], [(9, 1, 1)], direction=1, seed=1, compare_ref=False)
    check_c2c(dtype, [(30030, 1, 1)], [(2, 30030, 30030)], seed=2, compare_ref=False)
    for n in (6, 15, 98, 480):
        check_real(dtype, (n,), batch=5, compare_ref=False)


@pytest.mark.parametrize("n,b", [(1000, 50), (4096, 16), (10007, 8), (65521, 4), (120000, 4)])
def test_execute_captured_into_a_graph(n, b):
    """Launches with programmatic edges, between kernels of the caller, replay to the bytes of the direct call."""
    import torch
    lib = aoclfftz_b200.load()
    x = torch.from_numpy(synthetic.complex_uniform(n, n * b, np.complex64)).cuda()
    y, z = torch.empty_like(x), torch.empty_like(x)
    s = torch.cuda.Stream()
    plans = []
    for i, o, d in ((x, y, 0), (y, z, 1)):
        desc, _keep = abi.make_desc(i.data_ptr(), o.data_ptr(), [(n, 1, 1)], [(b, n, n)], 0, d, 1)
        plans.append(abi.setup(lib, desc, "f32"))
        assert plans[-1] and lib.aoclfftz_gpu_set_stream(plans[-1], s.cuda_stream) == 0
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(s):
            assert [lib.aoclfftz_execute(p) for p in plans] == [0, 0]
            s.synchronize()
            direct = z.clone()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                y.zero_()
                assert [lib.aoclfftz_execute(p) for p in plans] == [0, 0]
                twice = z * 2
            for _ in range(3):
                z.zero_()
                g.replay()
        torch.cuda.synchronize()
        assert torch.equal(z, direct) and torch.equal(twice, direct * 2)
        del g
    finally:
        for p in plans:
            lib.aoclfftz_destroy(p)

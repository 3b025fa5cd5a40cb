"""CPU check of the mixed-radix tile (csrc/kernels/fft_mr.cuh): the planner's
launch shape (fz_mr_shape, called in the built library) drives a restatement of
the kernel's index maps, slot by slot. Every stage has to touch each slot of its
lines exactly once and stay inside its shared memory, the reciprocals have to
divide exactly, and the tile's result has to be numpy's FFT."""
import ctypes as C

import numpy as np
import pytest

import aoclfftz_b200

I32, I64, U32, VP = C.c_int32, C.c_int64, C.c_uint32, C.c_void_p
MAXS, MAXB, MRS = 12, 8, 8
VAR_MR, F_TW4, F_MID = 11, 0x04, 0x40
IN_PAIRS, IN_SEPARATE = 1, 4  # fftz_in_kind


class Stage(C.Structure):
    _fields_ = [("r", I32), ("m", I32), ("nb", I32), ("tw", I32), ("mg_nb", U32), ("mg_m", U32), ("mg_b", U32),
                ("mg_r", U32)]


class Mr(C.Structure):
    _fields_ = [("st", Stage * MRS), ("pad", I32), ("mg_tpc", U32), ("big", I32), ("mg_pair", U32)]


class Pass(C.Structure):
    """fftz_pass_t (csrc/kernels/fftz_kernels.h)."""
    _fields_ = [("n", I32), ("nstages", I32), ("radix", I32 * MAXS), ("tw_off", I32 * MAXS), ("tpt", I32), ("tpc", I32),
                ("sstride", I32), ("nload", I32), ("nstore", I32), ("in_kind", I32), ("out_kind", I32), ("in_mode", I32),
                ("out_mode", I32), ("flags", I32), ("variant", I32),
                ("dtype", I32), ("nbdims", I32), ("ies", I64), ("oes", I64), ("ntf", I64), ("bdim", I64 * MAXB),
                ("ibs", I64 * MAXB), ("obs", I64 * MAXB), ("tw4_n", I64), ("tw4_l", I64), ("pre_n", I64),
                ("pre_es", I64), ("pre_cs", I64), ("post_n", I64), ("post_es", I64), ("post_cs", I64), ("mid_cs", I64),
                ("in_", VP), ("out", VP), ("tw", VP), ("tw4_hi", VP), ("tw4_lo", VP),
                ("pre_tab", VP), ("post_tab", VP), ("mid_tab", VP), ("rtw", VP), ("src_buf", I32), ("dst_buf", I32),
                ("ind_dim", I32), ("use_tma", I32), ("smem_tw", I32), ("test_tx_short", I32), ("ind_in", VP),
                ("ind_out", VP), ("mr", Mr), ("threads", I32), ("ntw", I32), ("pad2_", I32 * 6)]


def shape(n, dtype=0, col=False, two=False, tw4=False, ntf=100000, tpc=0, threads=0, cap=0, in_kind=0):
    lib = aoclfftz_b200.load()
    lib.fftz_pass_smem_bytes.restype = I64
    lib.fftz_smem_limit.restype = I64
    p = Pass(n=n, dtype=dtype, ntf=ntf, in_kind=in_kind, in_mode=int(col), out_mode=int(col), nbdims=1,
             flags=(F_MID if two else 0) | (F_TW4 if tw4 else 0))
    assert lib.fz_mr_shape(C.byref(p), tpc, threads, I64(cap or lib.fftz_smem_limit())) == 0
    assert p.variant == VAR_MR and 1 <= p.tpc <= ntf and 1 <= p.threads <= lib.fftz_mr_max_threads(dtype, p.mr.big)
    assert lib.fftz_pass_smem_bytes(C.byref(p)) <= lib.fftz_smem_limit()
    assert int(np.prod(p.radix[: p.nstages])) == n
    assert [(st.r, st.nb) for st in p.mr.st[: p.nstages]] == [(R, n // R) for R in p.radix[: p.nstages]]
    return p


def div(x, m):
    return (x.astype(np.uint64) * np.uint64(m) >> np.uint64(32)).astype(np.int64) if m else x


def exact_div(x, m, d):
    q = div(x, m)
    assert np.array_equal(q, x // d)
    return q


def items(p, s, col):
    """(line, position) of every item of a boundary stage."""
    nb = p.n // p.radix[s]
    i = np.arange(p.tpc * nb)
    if col:
        x = exact_div(i, p.mr.mg_tpc, p.tpc)
        return i - x * p.tpc, x
    q = exact_div(i, p.mr.st[s].mg_nb, nb)
    return q, i - q * nb


def mid_slots(p, s):
    R, M = p.radix[s], p.mr.st[s].m
    nb = p.n // R
    i = np.arange(p.tpc * nb)
    q = exact_div(i, p.mr.st[s].mg_nb, nb)
    j = i - q * nb
    b = exact_div(j, p.mr.st[s].mg_m, M)
    B = int(np.prod(p.radix[1:s]))
    return q * p.sstride + j + b * M * (R - 1) + exact_div(b, p.mr.st[s].mg_b, B) * p.mr.pad, j - b * M


def last_slots(p, line, K):
    o, q = np.zeros_like(K), K
    for s in range(p.nstages - 1):
        R, M = p.radix[s], p.mr.st[s].m
        nxt = exact_div(q, p.mr.st[s].mg_r, R)
        o, q = o + (q - nxt * R) * (M + p.mr.pad if s == 0 else M), nxt
    return line * p.sstride + o


def twiddle(R, M, rest):
    return np.exp(-2j * np.pi * np.outer(np.arange(R), rest) / (R * M))


def dft(v):
    return np.fft.fft(v, axis=0)


def check_slots(p, slots):
    assert slots.min() >= 0 and slots.max() < p.tpc * p.sstride
    assert np.unique(slots).size == slots.size == p.tpc * p.n


def simulate(p, x, mid=None):
    S, n = p.nstages, p.n
    sd = np.full(p.tpc * p.sstride, np.nan + 0j)
    y = np.full((p.tpc, n), np.nan + 0j)
    R, M = p.radix[0], n // p.radix[0]
    r = np.arange(R)[:, None]
    if S == 1:  # a thread a line: inputs and outputs 0 + r
        assert R == n and M == 1
        line = np.arange(p.tpc)
        y[line, r] = dft(x[line, r])
        return y
    line, rest = items(p, 0, p.in_mode)
    v = dft(x[line, rest + r * M]) * twiddle(R, M, rest)
    first = line * p.sstride + rest + r * (M + p.mr.pad)
    check_slots(p, first)
    sd[first] = v
    for s in range(1, S - 1):
        Rs, Ms = p.radix[s], p.mr.st[s].m
        base, rs = mid_slots(p, s)
        a = base + np.arange(Rs)[:, None] * Ms
        check_slots(p, a)
        sd[a] = dft(sd[a]) * twiddle(Rs, Ms, rs)
    Rl = p.radix[S - 1]
    nb = n // Rl
    line, K = items(p, S - 1, p.out_mode if mid is None else 0)
    a = last_slots(p, line, K) + np.arange(Rl)[:, None]
    check_slots(p, a)
    v = dft(sd[a])
    if mid is None:
        y[line, K + np.arange(Rl)[:, None] * nb] = v
        return y
    sd[a] = dft(np.conj(v) * mid[K + np.arange(Rl)[:, None] * nb])
    for s in range(S - 2, 0, -1):
        Rs, Ms = p.radix[s], p.mr.st[s].m
        base, rs = mid_slots(p, s)
        a = base + np.arange(Rs)[:, None] * Ms
        sd[a] = dft(sd[a] * twiddle(Rs, Ms, rs))
    line, rest = items(p, 0, p.out_mode)
    v = dft(sd[line * p.sstride + rest + r * (M + p.mr.pad)] * twiddle(R, M, rest))
    y[line, rest + r * M] = v
    return y


# one-stage lines, two to five stages, every radix, odd and even, the longest of each dtype
SIZES = [3, 11, 13, 14, 15, 16, 18, 35, 77, 100, 169, 360, 375, 1000, 1080, 1920, 2187, 2401, 4096, 11011, 14400, 15625,
         28000, 28800]


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_tile_is_the_transform(n, dtype, col):
    lib = aoclfftz_b200.load()
    if not lib.fz_mr_fits(dtype, I64(n), I64(227 * 1024)):
        assert n * (8 if dtype == 0 else 16) > 220 * 1024
        return
    p = shape(n, dtype, col)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((p.tpc, n)) + 1j * rng.standard_normal((p.tpc, n))
    y = simulate(p, x)
    ref = np.fft.fft(x, axis=1)
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [4, 6, 16, 40, 225, 2100, 20160])
def test_two_sweeps_are_the_convolution(n):
    p = shape(n, two=True)
    assert p.nstages >= 2
    rng = np.random.default_rng(n)
    x = rng.standard_normal((p.tpc, n)) + 1j * rng.standard_normal((p.tpc, n))
    mid = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ref = np.fft.fft(np.conj(np.fft.fft(x, axis=1)) * mid, axis=1)
    assert np.linalg.norm(simulate(p, x, mid) - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("ntf,tpc", [(1, 0), (3, 0), (5, 2), (700, 0), (100000, 3)])
def test_lines_per_cta_follow_the_batch_and_the_hint(ntf, tpc):
    p = shape(360, ntf=ntf, tpc=tpc, tw4=True)
    if tpc:
        assert p.tpc == min(tpc, ntf)
    else:
        assert p.tpc == 1 or ntf // p.tpc >= 296


def smooth13(n):
    for q in (2, 3, 5, 7, 11, 13):
        while n % q == 0:
            n //= q
    return n == 1


@pytest.mark.parametrize("dtype", [0, 1])
def test_a_tile_holds_several_lines_where_two_fit(dtype):
    """Column maps, real lines and lines-per-CTA hints of every length: a tile whose first choice of lines does not fit
    takes the next smaller one, with a block of its own, not one line on a single warp."""
    lib = aoclfftz_b200.load()
    lib.fz_ragged_smem_cap.restype = I64
    whole, share = 227 * 1024, lib.fz_ragged_smem_cap(dtype)
    for n in filter(smooth13, range(2, 29000)):
        line = (n + 32) * (8 << dtype) + 32
        if 2 * line > whole or not lib.fz_mr_fits(dtype, I64(n), I64(whole)):
            continue
        for kw in (dict(col=True), dict(tpc=4), dict(tpc=8), dict(col=True, in_kind=IN_PAIRS),
                   dict(col=True, in_kind=IN_SEPARATE)):
            p = shape(n, dtype, ntf=4096, **kw)
            assert p.tpc > 1 and p.threads >= 64, (n, kw)
        if 2 * (line + 16 * (8 << dtype)) <= share:
            for tw4 in (False, True):
                for ntf in (9, 20, 4096):
                    assert shape(n, dtype, col=True, tw4=tw4, ntf=ntf, threads=256, cap=share).tpc > 1, (n, tw4, ntf)


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("n,dtype", [(4840, 0), (5000, 0), (9000, 0), (12000, 0), (2560, 1), (3630, 1), (4840, 1), (5000, 1)])
def test_few_long_columns_spread_over_the_device(n, dtype, two):
    """Columns whose tile would fill an SM: where one round of CTAs takes them all, no more a tile than that needs (a
    power of two); many rounds of tiles hold a power of two of columns."""
    for ntf in (1, 17, 64, 148):
        assert shape(n, dtype, col=True, two=two, ntf=ntf).tpc == 1, ntf
    assert shape(n, dtype, col=True, two=two, ntf=296).tpc <= 2
    p = shape(n, dtype, col=True, two=two, ntf=50000)
    assert p.tpc & (p.tpc - 1) == 0


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("n", [1000, 2100, 2197, 4096, 12000])
def test_a_lone_cta_is_not_a_small_one(n, dtype):
    """One line: no other CTA shares its SM, so its block covers at least half of a stage's butterflies (or of the largest
    block)."""
    lib = aoclfftz_b200.load()
    p = shape(n, dtype, ntf=1)
    most = lib.fftz_mr_max_threads(dtype, p.mr.big)
    assert 2 * p.threads >= min(most, max(st.nb for st in p.mr.st[: p.nstages]))


@pytest.mark.parametrize("n,dtype,ntf,least", [(2, 0, 5000, 64), (144, 0, 40, 14), (5250, 0, 3, 1), (5600, 1, 2, 1), (1, 0, 9, 1)])
def test_executor_tiles_keep_their_block_and_share(n, dtype, ntf, least):
    """The ragged executor's tiles: 256 threads, within its share of shared memory, small batches not cut up."""
    lib = aoclfftz_b200.load()
    lib.fz_ragged_smem_cap.restype = I64
    cap = lib.fz_ragged_smem_cap(dtype)
    p = shape(n, dtype, ntf=ntf, threads=256, cap=cap)
    assert p.threads == 256 and lib.fftz_pass_smem_bytes(C.byref(p)) <= cap
    assert least <= p.tpc <= ntf


def pair_items(p, s):
    """(line, butterfly, mirrored butterfly) of every item of the stage that holds mirrored butterflies."""
    nb = p.n // p.radix[s]
    items_ = (nb + 1) // 2
    i = np.arange(p.tpc * items_)
    if p.in_mode:
        q = exact_div(i, p.mr.mg_tpc, p.tpc)
        line = i - q * p.tpc
    else:
        line = exact_div(i, p.mr.mg_pair, items_)
        q = i - line * items_
    return line, q, np.where(q > 0, nb - q, 0 if nb & 1 else nb // 2)


def half_spectrum_pairs(nb, R):
    """mr_store_half / mr_load_half: (butterfly and value of bin k, of bin n - k, k) of every pair that an item q holds;
    butterfly 0 is A (bins q + r nb), 1 is B (its mirror)."""
    def pairs(q):
        if q:
            return [((0, r), (1, R - 1 - r), q + r * nb) for r in range(R)]
        out = [((0, r), (0, (R - r) % R), r * nb) for r in range(R // 2 + 1)]
        if nb % 2 == 0:
            out += [((1, r), (1, R - 1 - r), nb // 2 + r * nb) for r in range((R - 1) // 2 + 1)]
        return out
    return pairs


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("n", [1, 2, 7, 13, 15, 16, 18, 25, 77, 121, 143, 240, 256, 1000, 1024, 2401, 22050])
def test_mirrored_butterflies_cover_each_bin_once(n, col):
    """r2c / c2r: the paired stage's items hold every butterfly of every line once, and the pairs of bins k, n - k that they
    recombine (separate) are every bin of the half spectrum (every value of the packed line) once, with numpy's result; the
    stage's radix is one its two-butterfly form exists for."""
    rng = np.random.default_rng(n)
    for kind in (IN_PAIRS, IN_SEPARATE):
        p = shape(n, col=col, in_kind=kind)
        s = p.nstages - 1 if kind == IN_PAIRS else 0
        R, nb = p.radix[s], n // p.radix[s]
        assert p.nstages == 1 or R <= 8 or R in (11, 13)
        if p.nstages == 1:
            line, a, b = np.arange(p.tpc), np.zeros(p.tpc, int), np.zeros(p.tpc, int)
        else:
            line, a, b = pair_items(p, s)
        own = np.concatenate([line * nb + a, (line * nb + b)[a != b]])
        assert np.array_equal(np.sort(own), np.arange(p.tpc * nb))
        x = rng.standard_normal(2 * n)
        Z, X = np.fft.fft(x[0::2] + 1j * x[1::2]), np.fft.rfft(x)
        w = np.exp(-1j * np.pi * np.arange(n + 1) / n)
        bins, vals = np.full(n + 1, np.nan + 0j), np.full(n, np.nan + 0j)
        pairs = half_spectrum_pairs(nb, R)
        for q, m in {(int(q), int(m)) for q, m in zip(a, b)}:
            at = {0: q, 1: m}
            for (f, r), (g, t), k in pairs(q):
                i, j = at[f] + r * nb, at[g] + t * nb
                assert i == k and j == (n - k) % n
                if kind == IN_PAIRS:
                    E, O = (Z[i] + np.conj(Z[j])) / 2, -0.5j * (Z[i] - np.conj(Z[j]))
                    assert np.isnan(bins[k]) and (k == n - k or np.isnan(bins[n - k]))
                    bins[k], bins[n - k] = E + w[k] * O, np.conj(E - w[k] * O)
                else:
                    S, D = X[k] + np.conj(X[n - k]), np.conj(w[k]) * (X[k] - np.conj(X[n - k]))
                    assert np.isnan(vals[i]) and (i == j or np.isnan(vals[j]))
                    vals[j], vals[i] = np.conj(S) + 1j * np.conj(D), S + 1j * D
        if kind == IN_PAIRS:
            assert np.linalg.norm(bins - X) <= 1e-13 * np.linalg.norm(X)
            if p.nstages > 1:
                y = rng.standard_normal((p.tpc, n)) + 0j
                assert np.linalg.norm(simulate(p, y) - np.fft.fft(y, axis=1)) <= 1e-13 * np.linalg.norm(y) * np.sqrt(n)
        else:
            assert np.linalg.norm(vals - 2 * Z) <= 1e-13 * np.linalg.norm(Z) * 2


class Blob(C.Structure):
    """fz_blob (csrc/host/fz_internal.h)."""
    _fields_ = [("p", VP), ("len", C.c_size_t), ("cap", C.c_size_t)]


@pytest.mark.parametrize("form,parts,eps", [(0, 1, 2.0 ** -24), (1, 1, 2.0 ** -53), (2, 2, 2.0 ** -63)])
@pytest.mark.parametrize("N", [1, 6, 4096, 120000, 3 * 2 ** 20 + 1])
def test_four_step_factor_tables(N, form, parts, eps):
    """W_N^r = hi[r / L] lo[r % L] for every r, each entry rounded once: floats, doubles, or a sum of two doubles (whose
    second is what the first left, down to the long double it was formed in)."""
    lib = aoclfftz_b200.load()
    b, L, hi, lo = Blob(), I64(), I64(), I64()
    assert lib.fz_tw4_tables(C.byref(b), form, I64(N), C.byref(L), C.byref(hi), C.byref(lo)) == 0
    raw = (C.c_ubyte * b.len).from_address(b.p)
    real = np.float32 if form == 0 else np.float64

    def entries(off, n):
        v = np.frombuffer(raw, dtype=real, count=2 * parts * n, offset=off).astype(np.longdouble).reshape(n, parts, 2)
        return v.sum(axis=1)

    nhi = -(-N // L.value)
    h, l = entries(hi.value, nhi), entries(lo.value, L.value)
    for got, r in ((h, np.arange(nhi) * L.value), (l, np.arange(L.value))):
        a = 2 * np.arctan2(np.longdouble(0), np.longdouble(-1)) * r.astype(np.longdouble) / N
        # half a unit in the last place of a value below one, plus this angle's own error: up to 2 pi in long double, its
        # pi, product and quotient each rounded by at most 2^-62, and the cosine
        assert np.abs(got - np.stack([np.cos(a), -np.sin(a)], axis=1)).max() <= eps / 2 + 4 * 2.0 ** -62
    assert b.len >= lo.value + L.value * parts * 2 * real().itemsize


@pytest.mark.parametrize("n1,n2,R", [(375, 320, 15), (16, 5000, 4), (1331, 121, 11)])
def test_four_step_factors_of_a_butterfly(n1, n2, R):
    """mr_store: output K + r nb of column c times W^{c K} W^{c nb r}, both factors found below N in the tables."""
    lib = aoclfftz_b200.load()
    N, nb = n1 * n2, n1 // R
    b, L, hi, lo = Blob(), I64(), I64(), I64()
    assert lib.fz_tw4_tables(C.byref(b), 1, I64(N), C.byref(L), C.byref(hi), C.byref(lo)) == 0
    raw = (C.c_ubyte * b.len).from_address(b.p)
    h = np.frombuffer(raw, dtype=np.complex128, count=-(-N // L.value), offset=hi.value)
    l = np.frombuffer(raw, dtype=np.complex128, count=L.value, offset=lo.value)
    assert L.value & (L.value - 1) == 0  # found by a shift and a mask
    c, K, r = np.meshgrid(np.arange(0, n2, 7), np.arange(nb), np.arange(R), indexing="ij")

    def factor(e):
        assert e.max() < N
        return h[e // L.value] * l[e % L.value]

    exact = np.exp(-2j * np.pi * (c * (K + r * nb)) / N)
    # three products of values of modulus 1, each part rounded once, and exp's own angle of up to 2 pi
    assert np.abs(factor(c * K) * factor(c * nb * r) - exact).max() <= 16 * 2.0 ** -52


def test_four_step_factors_beyond_32_bits_are_refused():
    lib = aoclfftz_b200.load()
    b, L, hi, lo = Blob(), I64(), I64(), I64()
    assert lib.fz_tw4_tables(C.byref(b), 1, I64(1 << 32), C.byref(L), C.byref(hi), C.byref(lo)) != 0
    assert not b.p


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("n,m", [(3, 6), (17, 35), (17, 36), (101, 210), (101, 224), (521, 1125), (2053, 5145),
                                 (2053, 4320), (5003, 10240), (16411, 53760), (40009, 81920)])
def test_chirp_tables(n, m, dtype):
    """The chirps and the convolution spectrum over m against long double: each part rounded once to the working
    precision (rel. error of a complex value at most eps / 2), in double plans beyond 65536 points formed in double,
    whose FFT adds at most eps a bit."""
    import scipy.fft
    lib = aoclfftz_b200.load()
    eps = 2.0 ** (-23 if dtype == 0 else -52)
    ct = np.complex64 if dtype == 0 else np.complex128
    j = np.array([k * k % (2 * n) for k in range(n)]).astype(np.longdouble)
    ang = j * 4 * np.arctan(np.longdouble(1)) / n
    c = np.cos(ang) - 1j * np.sin(ang)
    b = np.zeros(m, dtype=np.clongdouble)
    b[:n] = np.conj(c)
    b[m - np.arange(1, n)] = np.conj(c[1:])
    for direction in (0, 1):
        blob, offs = Blob(), [I64() for _ in range(3)]
        assert lib.fz_bluestein_tables(C.byref(blob), dtype, I64(n), I64(m), direction, *[C.byref(o) for o in offs]) == 0
        raw = (C.c_ubyte * blob.len).from_address(blob.p)
        pre, post, mid = [np.frombuffer(raw, dtype=ct, count=k, offset=o.value) for k, o in zip((n, n, m), offs)]
        for got, ref, bits in ((pre, c, 0), (post, c if direction == 0 else np.conj(c), 0),
                               (mid, np.conj(scipy.fft.fft(b)) / m, np.log2(m) if dtype == 1 and m > 65536 else 0)):
            err = np.linalg.norm((got - ref).astype(np.complex128)) / np.linalg.norm(ref.astype(np.complex128))
            assert err <= (0.5 + bits) * eps

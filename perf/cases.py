"""The workloads this library is timed on, each run through its C ABI (ctypes).

A case is a dict of plain values:
  kind    "c2c", "real" (r2c forward / c2r backward), "ragged" (many lengths in one
          launch) or "host" (c2c on page-locked host buffers, staged by the library)
  dims    transform sizes, innermost first, as text: "4096", "1920x1080"
  batch   transforms per call
  dtype   "f32" or "f64"
  step    "forward", "backward" or "both" (forward, then backward on its result)
  place   "out" of place, or "in" place (the data arrives in the buffer by a copy,
          since a transform overwrites it)
  layout  "rows" (each transform contiguous) or "columns" (1-D, neighbouring
          transforms one element apart)
Ragged batches have count / lo / hi / lengths (the seed of the lengths) instead of
dims and batch: lengths log-uniform in [lo, hi], one third each powers of two,
7-smooth numbers and primes, as in the library's own benchmark.

Transforms are unnormalised in both directions. Inputs are U[-1, 1) for complex
signals and N(0, 1) for ragged batches and real fields, made on the GPU from the seed.
"""
import ctypes as C
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aocl-fftz_b200", "python"))

import aoclfftz_b200  # noqa: E402
from aoclfftz_b200 import abi, synthetic  # noqa: E402

REAL = {"f32": torch.float32, "f64": torch.float64}
CPLX = {"f32": torch.complex64, "f64": torch.complex128}


def c2c(name, dims, batch, dtype="f32", step="both", place="out", layout="rows", kind="c2c"):
    return {"name": name, "kind": kind, "dims": dims, "batch": batch, "dtype": dtype, "step": step, "place": place,
            "layout": layout}


def listed():
    return [
        # a few short spectra inside a control or signal loop: the call itself is the cost
        c2c("tiny_f32", "512", 4),
        # the library's first benchmark shape: a batch of 4096-point lines, forward then backward
        c2c("rows4096_f32", "4096", 1024),
        # the headline benchmark: four lines of 2^24 points, forward then backward
        c2c("fourstep24_f32", str(1 << 24), 4),
        # a large batch of short mixed-radix lines (the benchmark's N = 1000 = 2^3 5^3)
        c2c("mixed1000_f32", "1000", 32768),
        # long lines of a sampling-rate length, 120000 = 2^6 3 5^4, in double
        c2c("smooth120000_f64", "120000", 64, "f64", "forward"),
        # a length nobody chose: prime, so a chirp-z transform
        c2c("prime10007_f32", "10007", 512, "f32", "backward"),
        # the ragged benchmark: 4096 transforms of mixed lengths in one launch
        {"name": "ragged_f32", "kind": "ragged", "count": 4096, "lo": 2, "hi": 65536, "lengths": 1, "dtype": "f32",
         "step": "both"},
        # a smaller ragged batch in double, one direction
        {"name": "ragged_f64", "kind": "ragged", "count": 1024, "lo": 2, "hi": 65536, "lengths": 2, "dtype": "f64",
         "step": "backward"},
        # a real field on a 512^3 grid in double, to the spectrum and back (a spectral solver's step)
        c2c("real3d512_f64", "512x512x512", 1, "f64", "both", kind="real"),
        # short frames of a real signal, to the spectrum and back
        c2c("frames2048_f32", "2048", 8192, "f32", "both", kind="real"),
        # four 1920 x 1080 images, transformed in the buffer they are loaded into
        c2c("image_f32", "1920x1080", 4, "f32", "forward", "in"),
        # the same 4096-point batch from and to host memory, as a program written for the CPU library calls it
        c2c("host4096_f32", "4096", 1024, kind="host"),
    ]


# ------------------------------------------------------------------- drawn cases


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _prime(n):
    return n > 1 and all(n % f for f in range(2, math.isqrt(n) + 1))


def _length(rng, lo, hi, cls):
    """A length log-uniform in [lo, hi]: the next power of two, 7-smooth number or prime below it, or any."""
    n = max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    if cls == "pow2":
        return 1 << (n.bit_length() - 1)
    while (cls == "smooth" and not _smooth(n)) or (cls == "prime" and not _prime(n)):
        n -= 1
    return max(2, n)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))


def draw(rng):
    kind = rng.choices(["line", "grid", "real", "ragged", "host"], [45, 15, 20, 15, 5])[0]
    dtype = rng.choice(["f32", "f32", "f64"])
    step = rng.choice(["forward", "backward", "both"])
    if kind == "ragged":
        return {"kind": "ragged", "count": _logint(rng, 32, 2048), "lo": 2, "hi": rng.choice([2048, 16384, 65536]),
                "lengths": rng.randrange(1 << 20), "dtype": dtype, "step": step}
    cls = rng.choice(["pow2", "smooth", "smooth", "prime"])
    most = 1 << (22 if cls == "prime" else 24)
    if dtype == "f64":
        most //= 2
    if kind == "grid" or (kind == "real" and rng.random() < 0.4):
        rank = rng.choice([2, 3])
        top = 4096 if rank == 2 else 256
        dims = [_length(rng, 16, top, rng.choice(["pow2", "smooth", cls])) for _ in range(rank)]
        while math.prod(dims) > most:
            dims[dims.index(max(dims))] //= 2
    else:
        dims = [_length(rng, 4, min(most, 1 << 22) if kind != "host" else 65536, cls)]
    total = math.prod(dims)
    batch = max(1, _logint(rng, max(total, 256), max(most, total)) // total)
    if kind == "real":
        return c2c_drawn("real", dims, batch, dtype, step, "out", "rows")
    if kind == "host":
        return c2c_drawn("host", dims, min(batch, max(1, (1 << 22) // total)), dtype, step, "out", "rows")
    place = "in" if rng.random() < 0.25 else "out"
    layout = "columns" if kind == "line" and batch > 1 and rng.random() < 0.3 else "rows"
    return c2c_drawn("c2c", dims, batch, dtype, step, place, layout)


def c2c_drawn(kind, dims, batch, dtype, step, place, layout):
    case = c2c("", "x".join(map(str, dims)), batch, dtype, step, place, layout, kind)
    del case["name"]
    return case


# --------------------------------------------------------------------- the calls


class Plan:
    """A handle of the library, destroyed with the program's last reference to it."""

    def __init__(self, lib, handle):
        if not handle:
            raise RuntimeError("setup failed: %s" % lib.aoclfftz_gpu_last_error().decode())
        self.lib, self.handle = lib, handle

    def __del__(self):
        if self.handle:
            self.lib.aoclfftz_destroy(self.handle)


def plan(src, dst, dims, vecs, case, direction):
    """A plan of aoclfftz_setup_* on these buffers; dims / vecs are (n, in stride, out stride)."""
    lib = aoclfftz_b200.load()
    desc, _keep = abi.make_desc(src.data_ptr(), dst.data_ptr(), dims, vecs, 1 if case["kind"] == "real" else 0, direction,
                                0 if src.data_ptr() == dst.data_ptr() else 1)
    return Plan(lib, abi.setup(lib, desc, case["dtype"]))


def sizes_of(case):
    if case["kind"] == "ragged":
        return synthetic.ragged_sizes(case["lengths"], case["count"], case["lo"], case["hi"])
    return [int(n) for n in case["dims"].split("x")]


def directions(case):
    return {"forward": [0], "backward": [1], "both": [0, 1]}[case["step"]]


def strides(sizes, first=None):
    """(n, stride) per dimension of a dense array, innermost first; `first`: its length in memory."""
    out, s = [], 1
    for i, n in enumerate(sizes):
        out.append((n, s))
        s *= first if i == 0 and first else n
    return out, s


def signal(case, seed):
    """The call's input in double on the GPU: complex [batch, ..., n1, n0] or real (for r2c, and before c2r)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "ragged":
        total = sum(sizes_of(case))
        return torch.view_as_complex(torch.randn(total, 2, generator=g, device="cuda", dtype=torch.float32)).to(
            torch.complex128)
    shape = [case["batch"]] + sizes_of(case)[::-1]
    if case["kind"] == "real":
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).double()
    x = torch.rand(shape + [2], generator=g, device="cuda", dtype=torch.float32)
    return torch.view_as_complex(x.double() * 2 - 1)


def given(case, seed):
    """What the program holds before the call, in its own precision (see signal)."""
    x = signal(case, seed)
    if case["kind"] != "real":
        return x.to(CPLX[case["dtype"]])
    if directions(case)[0] == 0:
        return x.to(REAL[case["dtype"]])
    axes = list(range(1, x.dim()))
    return torch.fft.rfftn(x, dim=axes, norm="ortho").to(CPLX[case["dtype"]])


def prepare(case, seed):
    x = given(case, seed)
    lib = aoclfftz_b200.load()
    dirs = directions(case)
    if case["kind"] == "ragged":
        sizes = sizes_of(case)
        arr = (C.c_int64 * len(sizes))(*sizes)
        bufs = [x] + [torch.empty_like(x) for _ in dirs]
        plans = [Plan(lib, lib.aoclfftz_gpu_ragged_setup(0 if case["dtype"] == "f32" else 1, d, len(sizes), arr, None,
                                                         None)) for d in dirs]
        return {"kind": "ragged", "plans": plans, "bufs": bufs}
    sizes, batch = sizes_of(case), case["batch"]
    if case["kind"] == "real":
        half = sizes[0] // 2 + 1
        rd, rspan = strides(sizes)
        hd, hspan = strides(sizes, half)
        real_shape = [batch] + sizes[::-1]
        half_shape = [batch] + ([half] + sizes[1:])[::-1]
        bufs, plans = [x], []
        for d in dirs:
            y = torch.empty(half_shape if d == 0 else real_shape, device="cuda",
                            dtype=(CPLX if d == 0 else REAL)[case["dtype"]])
            a, b, ia, ib = (rd, hd, rspan, hspan) if d == 0 else (hd, rd, hspan, rspan)
            plans.append(plan(bufs[-1], y, [(n, s, t) for (n, s), (_, t) in zip(a, b)], [(batch, ia, ib)], case, d))
            bufs.append(y)
        return {"kind": "real", "plans": plans, "bufs": bufs}
    if case["layout"] == "columns":
        x = x.reshape(batch, sizes[0]).t().contiguous()
        dims, vecs = [(sizes[0], batch, batch)], [(batch, 1, 1)]
    else:
        dd, span = strides(sizes)
        dims, vecs = [(n, s, s) for n, s in dd], [(batch, span, span)]
    if case["kind"] == "host":
        x = x.cpu().pin_memory()
        bufs = [x] + [torch.empty(x.shape, dtype=x.dtype).pin_memory() for _ in dirs]
    elif case["place"] == "in":
        bufs = [torch.empty_like(x)] * (len(dirs) + 1)
    else:
        bufs = [x] + [torch.empty_like(x) for _ in dirs]
    plans = [plan(bufs[i], bufs[i + 1], dims, vecs, case, d) for i, d in enumerate(dirs)]
    return {"kind": case["kind"], "plans": plans, "bufs": bufs, "new": x if case["place"] == "in" else None}


def run(state):
    plans, bufs = state["plans"], state["bufs"]
    if state["kind"] == "ragged":
        for i, p in enumerate(plans):
            if p.lib.aoclfftz_gpu_ragged_execute(p.handle, bufs[i].data_ptr(), bufs[i + 1].data_ptr()):
                raise RuntimeError(p.lib.aoclfftz_gpu_last_error().decode())
        return bufs[1:]
    if state.get("new") is not None:
        bufs[0].copy_(state["new"])
    for p in plans:
        if p.lib.aoclfftz_execute(p.handle):
            raise RuntimeError(p.lib.aoclfftz_gpu_last_error().decode())
    return bufs[-1:] if state.get("new") is not None else bufs[1:]


def work(case):
    sizes, dirs = sizes_of(case), directions(case)
    esz = 8 if case["dtype"] == "f32" else 16
    if case["kind"] == "ragged":
        return {"bytes": 2 * esz * sum(sizes) * len(dirs), "flops": sum(5 * n * math.log2(n) for n in sizes) * len(dirs)}
    total = case["batch"] * math.prod(sizes)
    flops = 5 * total * math.log2(math.prod(sizes)) * len(dirs)
    if case["kind"] == "real":
        half = total // sizes[0] * (sizes[0] // 2 + 1)
        return {"bytes": (total * esz // 2 + half * esz) * len(dirs), "flops": flops / 2}
    return {"bytes": 2 * esz * total * (1 if case["place"] == "in" else len(dirs)), "flops": flops}


def tolerance(case):
    # about four times the error against 64 bits measured on B200 (float 1e-7 ... 3.3e-7, double 3e-16 ... 7e-16)
    return {"rel": 2e-6 if case["dtype"] == "f32" else 4e-15}


def exact(case, seed):
    dirs = directions(case)
    x = given(case, seed)
    x = x.to(torch.complex128) if x.is_complex() else x.double()
    if case["kind"] == "ragged":
        sizes = sizes_of(case)
        offs, o = {}, 0
        for n in sizes:
            offs.setdefault(n, []).append(o)
            o += n
        y, z = torch.empty_like(x), torch.empty_like(x)
        for n, at in offs.items():
            ix = torch.tensor(at, device="cuda")[:, None] + torch.arange(n, device="cuda")
            line = x[ix]
            y[ix] = torch.fft.fft(line) if dirs[0] == 0 else torch.fft.ifft(line, norm="forward")
            z[ix] = line * n
        return [y, z] if len(dirs) == 2 else [y]
    axes = list(range(1, x.dim()))
    sizes = sizes_of(case)
    if case["kind"] == "real":
        if dirs[0] == 1:
            return [torch.fft.irfftn(x, s=sizes[::-1], dim=axes, norm="forward")]
        y = torch.fft.rfftn(x, dim=axes)
        return [y, x * math.prod(sizes)] if len(dirs) == 2 else [y]
    y = torch.fft.fftn(x, dim=axes) if dirs[0] == 0 else torch.fft.ifftn(x, dim=axes, norm="forward")
    outs = [y, x * math.prod(sizes)] if len(dirs) == 2 else [y]
    if case["place"] == "in":
        outs = outs[-1:]
    if case["layout"] == "columns":
        outs = [v.reshape(case["batch"], sizes[0]).t() for v in outs]
    return [v.cpu() for v in outs] if case["kind"] == "host" else outs

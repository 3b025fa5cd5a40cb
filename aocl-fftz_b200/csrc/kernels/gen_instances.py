#!/usr/bin/env python3
"""Writes the explicit instantiation files of the compile-time FFT kernels.

One file per (dtype, feature group) so that the build compiles them in parallel.
Each file exports a lookup  const void *fftz_fast_<dt>_<grp>(int log2n, int feat)
returning the kernel for that shape, or NULL.
"""
GROUPS = {
    "a": [(0, 1), (1, 5)],            # (FEAT, smallest log2 n): plain, four-step twiddle
    "c": [(16, 6), (17, 6)],          # pipelined (FEAT 16 + bits): plain, four-step twiddle
}
DTYPES = {"f32": ("float", 14), "f64": ("double", 13)}

for dt, (ctype, maxl) in DTYPES.items():
    for g, feats in GROUPS.items():
        lines = ["// GENERATED by gen_instances.py: compile-time FFT kernels, %s, group %s." % (ctype, g),
                 '#include "fft_fast.cuh"', "",
                 'extern "C" const void *fftz_fast_%s_%s(int log2n, int feat) {' % (dt, g),
                 "  switch (64 * feat + log2n) {"]
        for feat, lo in feats:
            kern = "fft_pipe_kernel" if feat >= 16 else "fft_fast_kernel"
            for l in range(lo, maxl + 1):
                lines.append("    case %d: return (const void *)&fftz::%s<%s, %d, %d>;"
                             % (64 * feat + l, kern, ctype, 1 << l, feat & 15))
        lines += ["    default: return 0;", "  }", "}", ""]
        open("fft_fast_%s_%s.cu" % (dt, g), "w").write("\n".join(lines))

#!/usr/bin/env python3
"""Writes csrc/dft_consts.cuh: cos/sin(2 pi m / R) for the odd prime DFT
lengths R in {3, 5, 11, 31}, evaluated in double precision and rounded once
to binary32.  And csrc/mixed_radix_consts.cuh: the same functions in both
precisions for the radices of the mixed-radix FFTs."""
import math
import os

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))


def fmt(v):
    return "%.9ef" % float(np.float32(v))


def main():
    out = ["// Generated constants: cos/sin(2*pi*m/R) rounded to float, R in {3,5,11,31}.",
           "// Produced by evaluating the trigonometric functions in double precision (Python math) and",
           "// rounding once to binary32 (tart-gnss_b200/gen_dft_consts.py).",
           "#pragma once", ""]
    for R in (3, 5, 11, 31):
        c = [math.cos(2 * math.pi * m / R) for m in range(R)]
        s = [math.sin(2 * math.pi * m / R) for m in range(R)]
        out.append("__constant__ float kCos%d[%d] = {%s};" % (R, R, ", ".join(fmt(v) for v in c)))
        out.append("__constant__ float kSin%d[%d] = {%s};" % (R, R, ", ".join(fmt(v) for v in s)))
    open(os.path.join(HERE, "csrc", "dft_consts.cuh"), "w").write("\n".join(out) + "\n")
    out = ["// Generated constants: cos/sin(2*pi*m/R) in double precision (Python math,",
           "// tart-gnss_b200/gen_dft_consts.py) and rounded once to float, for the radices of the", "// mixed-radix FFTs.",
           "#pragma once", ""]
    for R in (3, 5, 7, 11, 13, 25, 31, 32):
        for name, f in (("Cos", math.cos), ("Sin", math.sin)):
            v = [f(2 * math.pi * m / R) for m in range(R)]
            out.append("__constant__ double k%sD%d[%d] = {%s};" % (name, R, R, ", ".join(repr(x) for x in v)))
            out.append("__constant__ float k%sF%d[%d] = {%s};" % (name, R, R, ", ".join(fmt(x) for x in v)))
    open(os.path.join(HERE, "csrc", "mixed_radix_consts.cuh"), "w").write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()

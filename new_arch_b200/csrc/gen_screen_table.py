"""Writes scmf_screen_table.h: the piecewise-linear half-normal quantile of the
move kernel's screen (screen_normal in scmf_sweep.cuh).

The screen needs a normal only to within SCMF_SCREEN_DELTA: a trial that it
cannot reject with that error allowed for is proposed again with the exact
normals (normal_of).  Same argument as there: f = float(2 (w mod 2^31) + 1) in
[1, 2^32], h(v) = -Phi^-1(v / 2) at v = f 2^-32.  Four segments per binade of f,
picked by the top two mantissa bits: entry (bits(f) >> 21) - 127 * 4, 0 .. 128
(128 is f = 2^32 alone, h = 0).  Each is c0 + c1 f, the line of least largest
error over the segment (the chord of a convex function, lowered by half its
largest distance), scaled by 2^30 (see ScreenDev in scmf_internal.h).  The 513
cubic segments of the exact table take 8 KB a copy; these 129 pairs take 1 KB,
so that sixteen lane-interleaved copies fit beside the positions.

Run: python gen_screen_table.py > scmf_screen_table.h
"""
import sys

import numpy as np
from scipy.special import ndtri

from gen_normal_table import hexf

SEG_BITS = 2
N_SEG = 32 * (1 << SEG_BITS) + 1
SCALE = 2.0 ** 30
SAMPLES = 4097


def h(f):
    return -ndtri(np.asarray(f) * 2.0 ** -33)


def segment(idx):
    e, j = divmod(idx, 1 << SEG_BITS)
    f0 = 2.0 ** e * (1.0 + j / (1 << SEG_BITS))
    f1 = f0 + 2.0 ** (e - SEG_BITS)
    f = np.linspace(f0, f1, SAMPLES)
    slope = (h(f1) - h(f0)) / (f1 - f0)
    c1 = np.float32(slope * SCALE)
    rest = h(f) - float(c1) / SCALE * f
    c0 = np.float32(0.5 * (rest.max() + rest.min()) * SCALE)
    err = np.abs(h(f) - (float(c0) + float(c1) * f) / SCALE).max()
    return c0, c1, err


def table():
    tab, worst = np.zeros((N_SEG, 2), np.float32), 0.0
    for idx in range(N_SEG - 1):
        tab[idx, 0], tab[idx, 1], err = segment(idx)
        worst = max(worst, err)
    return tab, worst


def main(out=sys.stdout):
    tab, worst = table()
    delta = 1.05 * worst + 1e-5       # the exact table's own error and the rounding of c0 + c1 f
    out.write("/* Generated by gen_screen_table.py: piecewise-linear half-normal quantile,\n"
              " * 129 segments of (c0, c1) scaled by 2^30; see that script. */\n")
    out.write("#pragma once\n#define SCMF_SCREEN_SEGS %d\n#define SCMF_SCREEN_DELTA %.6e\n"
              "#define SCMF_SCREEN_TABLE_DATA \\\n" % (N_SEG, delta))
    out.write(", \\\n".join("    %s, %s" % (hexf(a), hexf(b)) for a, b in tab) + "\n")


if __name__ == "__main__":
    main()

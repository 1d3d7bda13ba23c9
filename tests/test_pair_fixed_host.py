"""The arithmetic of the fixed-point pair term on the host: csrc/co_pair_fixed.cuh compiles
there too (the device's seed of 1/sqrt is a correctly rounded one). 1/|d|^3 of normalised
distances against extended precision.

Tolerance: e is rounded to 2^-52 and enters with 3/2 (1.5 units of 2^-53), c to 2^-52 (1), the
polynomial's factor to 2^-30 of e (0.5); truncations of the 64-bit products 0.4: 3.4 units,
bound 4; the mean of the squares a third of that.
"""
from __future__ import annotations

import os
import subprocess

import build

SRC = r"""
#include <math.h>
#include <string.h>
#include <stdio.h>
#include <stdlib.h>
#include "co_pair_fixed.cuh"
typedef long double ld;
static double uniform(unsigned long long &s) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(s >> 11) * 0x1p-53;
}
static fx_limb limb(double x) { return fx_split((fx64)(x * 0x1p61)); }
static ld value(fx_limb a, int e) { return ldexpl((ld)a.h * 2147483648.0L + a.l, e); }
int main() {
    unsigned long long s = 1;
    double worst = 0, square = 0;
    const int n = 300000;
    for (int i = 0; i < n; i++) {
        double a = 0.5 + 0.5 * uniform(s), b = (2 * uniform(s) - 1) * (i % 2 ? 0.9999 : a);
        if (i % 5 == 0) b = copysign(a, b);                  // |d1| = |d2|
        if (i % 1000 == 0) { a = 0.5; b = 0.0; }
        if (uniform(s) < 0.5) a = -a;
        fx_limb d1 = limb(a), d2 = limb(b);
        if (i % 3) { const fx_limb t = d1; d1 = d2; d2 = t; }
        const ld x = value(d1, -61), y = value(d2, -61);
        const double e = (double)(value(fx_invcube(d1, d2), -58) * powl(x * x + y * y, 1.5L) - 1) * 0x1p53;
        worst = fmax(worst, fabs(e));
        square += e * e;
    }
    printf("%.4f %.4f\n", worst, sqrt(square / n));
}
"""


def test_inverse_cube(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(build.HERE, "csrc"), str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    worst, rms = map(float, subprocess.run([str(exe)], check=True, capture_output=True,
                                           text=True).stdout.split())
    assert worst <= 4.0 and rms <= 4.0 / 3

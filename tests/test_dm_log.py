"""The table logarithm of the gathers' epilogue (dm_log), point by point against the 64-bit-mantissa
logl, on the CPU: the header's function compiled for the host (the same operations, fma included).
Bound: 3/2 2^-52 max(1, |log x|), from two roundings of the sum (2^-53 of it each), ln 2's
(0.15 2^-52 of it), the table's entry (2^-55) and the series' end."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdft-dev_general_b200", "csrc")
SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "k_angular_mma.cuh"
using namespace mdft;
static double2 tab[kLogN];
static double worst;
static void check(double x) {
    const long double l = logl((long double)x), e = fabsl((long double)dm_log(x, tab) - l);
    const double r = (double)(e / (0x1p-52L * fmaxl(1.0L, fabsl(l))));
    if (!(r <= worst)) worst = r;
}
int main() {
    dm_log_table(tab);
    // every table interval, in every binade from the smallest normal to the largest: its ends, the
    // neighbours of its ends, its middle and pseudo-random points
    unsigned long long seed = 20260101;
    for (int k = -1022; k <= 1023; ++k)
        for (int i = 0; i < kLogN; ++i) {
            const double lo = ldexp(1.0 + i / 128.0, k), hi = i + 1 < kLogN ? ldexp(1.0 + (i + 1) / 128.0, k) : nextafter(ldexp(1.0, k), 0) * 2;
            const double pts[] = {lo, nextafter(lo, hi), 0.5 * lo + 0.5 * hi, nextafter(hi, lo), hi};
            for (double x : pts) check(x);
            for (int j = 0; j < 8; ++j) {
                seed = seed * 6364136223846793005ull + 1442695040888963407ull;
                check(lo + (hi - lo) * ((seed >> 11) * 0x1p-53));
            }
        }
    // around one, where the logarithm is small
    for (int j = 1; j < 2000000; ++j) {
        check(1.0 + j * 0x1p-28);
        check(1.0 - j * 0x1p-28);
    }
    printf("%.17g %d %.17g\n", worst, dm_log(1.0, tab) == 0.0, dm_log(2.0, tab) - 0.69314718055994530942);
}
"""


def test_every_interval(tmp_path):
    src, exe = str(tmp_path / "log.cu"), str(tmp_path / "log")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["nvcc", "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", CSRC, "-o", exe, src])
    worst, one, two = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    print("\nlargest error: %s of 2^-52 max(1, |log x|)" % worst)
    assert float(worst) <= 1.5
    assert one == "1" and float(two) == 0.0

"""The reference's flush of R (src/module_energy_cproj_mrso.f90:491-492) against its form in the cell
records of k_ozc, which flush the factors e^{-i mu' alpha} and D: on the CPU, with the header's
recursion, over every cell of a grid.  The two agree but for entries that are small only as a
product, in each part within epsilon(1.) = 2^-23, none of them up to mmax 2 and below 1 in 1000."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdft-dev_general_b200", "csrc")
SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "common.cuh"
#include "setup_host.cuh"
#include "k_ozc.cuh"
using namespace mdft;
int main(int, char **v) {
    const int M = atoi(v[1]), n[3] = {atoi(v[2]), atoi(v[3]), atoi(v[4])};
    const double l[3] = {atof(v[5]), atof(v[6]), atof(v[7])};
    std::vector<int> xu;
    std::vector<double> cf;
    build_ozc_recipes(M, xu, cf);
    long total = 0, differ = 0;
    double worst = 0.0;
    for (int iz = 0; iz <= n[2] / 2; ++iz)
        for (int ib = 0; ib <= n[1] / 2; ++ib)
            for (int ia = 0; ia <= n[0] / 2; ++ia) {
                const double qx = ia * 2 * kPi / l[0], qy = ib * 2 * kPi / l[1], qz = iz * 2 * kPi / l[2];
                const double rho = std::sqrt(qx * qx + qy * qy), nrm = std::sqrt(qx * qx + qy * qy + qz * qz);
                const double ex = rho > 0 ? qx / rho : 1, ey = rho > 0 ? -qy / rho : 0;
                const double cb = nrm > 0 ? qz / nrm : 1, h = nrm > 0 ? rho / nrm * std::sqrt(0.5) : 0;
                std::vector<double> D(ozc_eoff(M + 1) + 16, 0.0);
                D[0] = 1;
                D[ozc_eidx(1, -1, 0)] = h;
                D[ozc_eidx(1, -1, 1)] = 0.5 * (1 - cb);
                D[ozc_eidx(1, 0, 0)] = cb;
                D[ozc_eidx(1, 0, 1)] = h;
                D[ozc_eidx(1, 1, 0)] = -h;
                D[ozc_eidx(1, 1, 1)] = 0.5 * (1 + cb);
                for (int k = 2; k <= M; ++k)
                    for (int e = ozc_eoff(k); e < ozc_eoff(k + 1); ++e) {
                        const int o = 3 * (e - ozc_eoff(2));
                        double s = 0;
                        for (int t = 0; t < 3; ++t) s += cf[o + t] * D[xu[o + t] & 0xffff] * D[xu[o + t] >> 16];
                        D[e] = s;
                    }
                double px = 1, py = 0;
                for (int k = 0; k <= M; ++k) {  // |mu'|
                    double sx = px, sy = py;
                    bool axis = k == 0;
                    if (std::fabs(px) < kEpsSp) { sx = 0; sy = py > 0 ? 1 : -1; axis = true; }
                    else if (std::fabs(py) < kEpsSp) { sx = px > 0 ? 1 : -1; sy = 0; axis = true; }
                    for (int lv = std::max(k, 1); lv <= M; ++lv)
                        for (int m = -k; m <= k; m += std::max(1, 2 * k))
                            for (int m1 = 0; m1 <= lv; ++m1, ++total) {
                                const double d = D[ozc_eidx(lv, m, m1)];
                                const double f = std::fabs(d) < kEpsSp ? 0 : axis ? (double)(float)d : d;
                                double re = px * d, im = py * d;  // the reference's product
                                if (std::fabs(re) < kEpsSp) { re = 0; im = (float)im; }
                                if (std::fabs(im) < kEpsSp) { re = (float)re; im = 0; }
                                const double e = std::max(std::fabs(sx * f - re), std::fabs(sy * f - im));
                                if (e > 1e-14) ++differ;
                                worst = std::max(worst, e);
                            }
                    const double x = px * ex - py * ey, y = px * ey + py * ex;
                    px = x;
                    py = y;
                }
            }
    printf("%ld %ld %.17g\n", total, differ, worst);
}
"""


@pytest.fixture(scope="module")
def emulate(tmp_path_factory):
    d = tmp_path_factory.mktemp("flush")
    src, exe = str(d / "flush.cu"), str(d / "flush")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["nvcc", "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", CSRC, "-o", exe, src])
    return exe


@pytest.mark.parametrize("mmax,dims,box", [(1, (96, 96, 96), (48, 48, 48)), (2, (24, 36, 48), (12, 18, 24)), (3, (64, 64, 64), (32, 32, 32)),
                                           (4, (32, 48, 24), (12, 19, 9.1)), (5, (32, 32, 32), (12, 12, 12)), (5, (64, 64, 64), (24, 24, 24))])
def test_flush_of_the_factors(emulate, mmax, dims, box):
    out = subprocess.run([emulate] + [str(x) for x in (mmax, *dims, *box)], capture_output=True, text=True, check=True).stdout
    total, differ, worst = (float(x) for x in out.split())
    print("\nmmax %d %s: %d of %d entries differ, by at most %.3e" % (mmax, dims, differ, total, worst))
    assert worst <= 2.0 ** -23
    assert differ <= (0 if mmax <= 2 else 1e-3 * total)

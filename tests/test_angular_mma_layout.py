"""Shared-memory layout of the projection on the matrix instructions (k_project_mma), on the CPU:
the shape arithmetic of the header, compiled for the host, over every angular order and symmetry
the engine accepts.  A stage is bm rows of 2 sa values; what the copies write of a row stays in it."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdft-dev_general_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "k_angular_mma.cuh"
using namespace mdft;
int main() {
    for (int mrso = 1; mrso <= 6; ++mrso)
        for (int M = 0; M <= kMaxMmax; ++M) {
            int np = 0;
            for (int m = 0; m <= M; ++m) np += (2 * m + 1) * (m / mrso + 1);
            const int no = (M + 1) * (2 * M + 1) * (2 * (M / mrso) + 1);
            const DmShape s = dm_project_shape<double>(np, no, 227 * 1024 - 1024);
            if (!s.nt) continue;
            int written = 0;
            for (int i = 0; i < s.nslab; ++i) {
                const int nu = (s.nkb - i * s.skb < s.skb ? s.nkb - i * s.skb : s.skb) * 4;
                const int n = dm_any_values(nu, s.sa);
                written = n > written ? n : written;
            }
            printf("%d %d %d %d %d %d %d %d %d %d %d %d %zu %d\n", M, mrso, no, s.bm, s.sa, s.pitch, s.nkb, s.skb, s.nstage, s.wn, s.nt, s.nb, s.smem, written);
        }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    src, exe = str(d / "layout.cu"), str(d / "layout")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, "-o", exe, src])
    names = ("mmax", "mrso", "no", "bm", "sa", "pitch", "nkb", "skb", "nstage", "wn", "nt", "nb", "smem", "written")
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return [dict(zip(names, map(int, line.split()))) for line in out.splitlines()]


def test_copies_of_an_unaligned_row_stay_in_it(shapes):
    assert any(2 * s["sa"] == s["no"] for s in shapes)  # unpadded rows are among them
    for s in shapes:
        assert s["written"] <= 2 * s["sa"], s
        assert s["written"] >= min(s["no"], 8 * s["skb"]), s


def test_a_stage_is_read_within_itself(shapes):
    # the last row of a tile reads 8 skb values from its start: within the stage and the pad after
    # it, which no copy reaches (the next stage may be in flight then)
    for s in shapes:
        assert (s["bm"] - 1) * s["sa"] + 4 * s["skb"] <= s["pitch"], s
        assert s["bm"] * s["sa"] <= s["pitch"], s
        # stages, the matrix, weights and the table fit in what is allocated
        need = 16 * (s["nstage"] * s["pitch"] + 4 * s["nkb"] * s["nb"])
        assert need <= s["smem"], s

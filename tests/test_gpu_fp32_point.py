"""Evaluations of an FP32 point (the FP32 phase of a mixed solve: FP32 point, potential, gradient
and direction) against the oracle, for every form of their kernels.

One iteration of the mixed minimiser without a polish moves the point by -df/|df| times the step,
so the evaluated gradient can be read off the move; the trace has F and max|df| of the start point
and F of the trial point, whose evaluation also forms df.d.  Bars, those of the mixed path:
F 2e-6 of |F|; the gradient 1e-4 of max|df|, to which the move adds the FP32 rounding of the start
and of the trial point (2^-24 of each) and of their difference's scale (FP32 df: 2^-23)."""
import re

import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine, PREC_MIXED
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT
EPS = 2.0 ** -24


def first_step(c, ck, vext, xi, capfd, **env):
    """(F at the start, max|df| there, F at the trial point, that point, forms) of one iteration."""
    with pytest.MonkeyPatch.context() as mp:
        for k in ("MDFT_ANGULAR", "MDFT_OZ"):
            mp.delenv(k, raising=False)
        for k, v in dict(env, MDFT_AUTOTUNE="0", MDFT_TRACE="1").items():
            mp.setenv(k, v)
        e = Engine(c["n"], c["L"], c["mmax"], ck, temperature=SV.temperature, n0=SV.n0, precision=PREC_MIXED)
    e.set_vext(vext)
    capfd.readouterr()
    x1, r = e.minimize(xi, m=5, pgtol=1e-12, ftol_abs=-1.0, itermax=1, precision=PREC_MIXED, polish=0)
    log = capfd.readouterr().err
    forms = e.kernel_forms()
    e.close()
    its = {int(i): (float(f), float(g)) for i, f, g in re.findall(r"mdft-trace it (\d+) nfg \d+ prec mixed f (\S+) gmax (\S+)", log)}
    assert r["iterations"] == 1 and r["evaluations_mixed"] >= 2 and sorted(its) == [0, 1], log
    assert "dN nan" in log  # the trace of an FP32 point
    return its[0][0], its[0][1], its[1][0], x1, forms


@pytest.mark.parametrize("name", ["mol8_m0", "ion16_m1", "mol16_m2", "mol24_m3"])
def test_fp32_point(tmp_path, name, capfd):
    c = cases.ALL_CASES[name]
    ck = cases.case_ck(tmp_path, c)
    o = O.Oracle(c["n"], c["L"], c["mmax"], ck, SV.kT, SV.n0)
    o.compute_vext(cases.solute_of(c), SV, rvdw=c["rvdw"])
    xi = cases.xi_of(c, o.shape)
    x0 = xi.astype(np.float32).astype(np.float64)
    fo, dfo, _ = o.energy_grad(x0)
    top = np.abs(dfo).max()
    modes = {"default": {}, "ffma": {"MDFT_ANGULAR": "ffma"}, "umma": {"MDFT_ANGULAR": "umma"},
             "ring": {"MDFT_ANGULAR": "ring"}, "ozp": {"MDFT_OZ": "ozp"}}
    moved = {}
    for mode, env in modes.items():
        f0, g0, f1, x1, forms = first_step(c, ck, o.get_vext(), xi, capfd, **env)
        assert forms["oz_factored"] == (mode != "ozp")
        assert not (mode in ("umma", "ffma") and (forms["gather_ring"] or forms["project_ring"]))
        assert not (mode == "ring" and not forms["project_ring"])
        assert abs(f0 - fo) <= 2e-6 * abs(fo), (mode, f0, fo)
        assert abs(g0 - top) <= 1e-4 * top, (mode, g0, top)
        move = x0 - x1
        scale = np.linalg.norm(dfo) / np.linalg.norm(move)  # the step's length cancels
        rounding = EPS * scale * (np.abs(x0) + np.abs(x1)) + 2 * EPS * np.abs(dfo)
        err = np.abs(move * scale - dfo)
        print("\n%s %s: F %.2e, df %.2e of max (bar %.2e)" % (name, mode, abs(f0 - fo) / abs(fo), err.max() / top,
                                                            1e-4 + rounding.max() / top))
        assert np.all(err <= 1e-4 * top + rounding), mode
        f1o, _, _ = o.energy_grad(x1)
        assert abs(f1 - f1o) <= 2e-6 * abs(f1o), (mode, f1, f1o)
        moved[mode] = x1
    # the forms are other kernels: their roundings differ (the ring and register ones share theirs)
    assert not np.array_equal(moved["ffma"], moved["umma"])
    if c["mmax"] > 0:
        assert not np.array_equal(moved["ozp"], moved["default"])

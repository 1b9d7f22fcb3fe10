"""The tables that only FP32 evaluations read are laid out before the first of them: a mixed
minimisation on an FP64 handle takes the same steps, bit for bit, as on a mixed handle (kernel
forms fixed), its FP64 evaluations are the same before and after it, and an FP64 handle that never
minimises in mixed precision holds less device memory."""
import numpy as np
import pytest
import torch

from mdft_b200 import Engine, PREC_FP64, PREC_MIXED
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("name,oz", [("mol8_m0", None), ("mol16_m2", None), ("mol16_m2", "ozp"), ("mol24_m3", None), ("rand8_m5", None)])
def test_mixed_minimisation_of_an_fp64_handle(tmp_path, name, oz, monkeypatch):
    c = cases.ALL_CASES[name]
    ck = cases.case_ck(tmp_path, c)
    monkeypatch.setenv("MDFT_AUTOTUNE", "0")
    if oz:
        monkeypatch.setenv("MDFT_OZ", oz)
    res = []
    for precision in (PREC_MIXED, PREC_FP64):
        with Engine(c["n"], c["L"], c["mmax"], ck, temperature=SV.temperature, n0=SV.n0, precision=precision) as e:
            sol = cases.solute_of(c)
            if sol is not None:
                e.compute_vext(sol, SV, rvdw=c["rvdw"])
            else:
                e.set_vext(cases.random_vext(c, e.shape))
            xi = cases.xi_of(c, e.shape)
            before = e.energy_and_gradient(xi) if precision == PREC_FP64 else None
            x, r = e.minimize(xi, m=5, pgtol=1e-9, ftol_abs=-1.0, itermax=6, precision=PREC_MIXED, polish=0)
            res.append((x, r))
            if before is not None:
                after = e.energy_and_gradient(xi)
                assert before[0] == after[0] and np.array_equal(before[1], after[1])
    assert np.array_equal(res[0][0], res[1][0]) and res[0][1] == res[1][1]
    assert res[0][1]["evaluations_mixed"] > 1


def test_memory_of_an_fp64_handle(tmp_path, monkeypatch):
    # 64^3 points: their FP32 cell records alone are 33 x 33 x 33 cells of 57 values at mmax 3
    c = cases.ALL_CASES["mol64_m3"]
    ck = cases.case_ck(tmp_path, c)
    monkeypatch.setenv("MDFT_AUTOTUNE", "0")

    def held(precision):
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        with Engine(c["n"], c["L"], c["mmax"], ck, temperature=SV.temperature, n0=SV.n0, precision=precision) as e:
            e.energy_and_gradient(np.ones(e.shape), want_grad=False)
            return free0 - torch.cuda.mem_get_info()[0]

    held(PREC_MIXED)  # modules and pools of the process
    mixed, fp64 = held(PREC_MIXED), held(PREC_FP64)
    assert mixed - fp64 >= 33 ** 3 * 57 * 4, (mixed, fp64)

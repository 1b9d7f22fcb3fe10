"""A solvent without a symmetry axis (mrso 1; the c(k) layouts hold it at mmax 0) against the oracle
in both precisions (F 1e-10 / 2e-6, gradient 1e-8 / 1e-4), and the two forms of the FP32 OZ step:
the factored one that the handle reports is another kernel than MDFT_OZ=ozp's."""
import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine, PREC_FP64, PREC_MIXED, synth
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("dims", [(16, 16, 16), (8, 12, 18)])
def test_mrso1(tmp_path, dims, monkeypatch):
    box = tuple(0.5 * n for n in dims)
    ck = synth.make_ck_file(str(tmp_path / "ck.txt"), 0, mrso=1, kmax=14.0, dk=0.05)
    o = O.Oracle(dims, box, 0, ck, SV.kT, SV.n0, mrso=1)
    rng = np.random.default_rng(dims[0])
    o.set_vext(0.8 * rng.standard_normal(o.shape))
    xi = 1.0 + 0.15 * rng.standard_normal(o.shape)
    f0, df0, t0 = o.energy_grad(xi)
    res = {}
    for name, precision, env in (("fp64", PREC_FP64, None), ("factored", PREC_MIXED, None), ("ozp", PREC_MIXED, "ozp")):
        if env:
            monkeypatch.setenv("MDFT_OZ", env)
        else:
            monkeypatch.delenv("MDFT_OZ", raising=False)
        monkeypatch.setenv("MDFT_AUTOTUNE", "0")
        with Engine(dims, box, 0, ck, temperature=SV.temperature, n0=SV.n0, mrso=1, precision=precision) as e:
            e.set_vext(o.get_vext())
            f1, df1, t1 = e.energy_and_gradient(xi)
            assert e.kernel_forms()["oz_factored"] == (env is None)
        etol, gtol = (1e-10, 1e-8) if precision == PREC_FP64 else (2e-6, 1e-4)
        assert abs(f1 - f0) <= etol * abs(f0) and np.all(np.abs(t1 - t0) <= etol * abs(f0)), (name, f1, f0)
        assert np.abs(df1 - df0).max() <= gtol * np.abs(df0).max(), name
        res[name] = df1
    assert not np.array_equal(res["factored"], res["ozp"])

"""FP64 evaluations where many entries of R are small (high angular order, more directions than the
small boxes of the other cases) against the oracle, which flushes R as the reference does: F, terms
and gradient at the FP64 bars (1e-10 of |F|, 1e-8 of max|df|), and the excess gradient alone."""
import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("mmax,dims,box", [(5, (32, 32, 32), (12.0, 12.0, 12.0)), (4, (32, 48, 24), (12.0, 19.0, 9.1)),
                                           (3, (64, 32, 96), (17.0, 9.0, 51.0))])
def test_small_entries_of_the_rotation(tmp_path, mmax, dims, box):
    ck = cases.ck_path(tmp_path, mmax, kmax=18.0, dk=0.05)
    o = O.Oracle(dims, box, mmax, ck, SV.kT, SV.n0)
    rng = np.random.default_rng(7 * mmax)
    o.set_vext(0.8 * rng.standard_normal(o.shape))
    xi = 1.0 + 0.15 * rng.standard_normal(o.shape)
    f0, df0, t0 = o.energy_grad(xi)
    rho = xi ** 2 * o.rho0
    w = o.weights
    dfid = np.where(rho > np.finfo(float).eps, w * 2 * o.rho0 * xi * (SV.kT * np.log(rho / o.rho0) + o.get_vext()), 0.0)
    exc0 = df0 - dfid
    with Engine(dims, box, mmax, ck, temperature=SV.temperature, n0=SV.n0) as e:
        e.set_vext(o.get_vext())
        f1, df1, t1 = e.energy_and_gradient(xi)
        exc1 = np.zeros(e.shape)
        e.excess_energy(xi, exc1)
    print("\nmmax %d: F %.2e, terms %.2e, df %.2e, excess df %.2e" % (
        mmax, abs(f1 - f0) / abs(f0), np.abs(t1 - t0).max() / abs(f0), np.abs(df1 - df0).max() / np.abs(df0).max(),
        np.abs(exc1 - exc0).max() / np.abs(exc0).max()))
    assert abs(f1 - f0) <= 1e-10 * abs(f0), (f1, f0)
    assert np.all(np.abs(t1 - t0) <= 1e-10 * abs(f0)), (t1, t0)
    assert np.abs(df1 - df0).max() <= 1e-8 * np.abs(df0).max()
    assert np.abs(exc1 - exc0).max() <= 1e-8 * np.abs(exc0).max()

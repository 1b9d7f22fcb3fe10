"""The OZ step by cells of points that share |q| and the polar angle (k_ozc), against the
oracle: every angular order, boxes whose cell count is not a multiple of a CTA's four, unequal
sides (frames with the azimuth on and off the axes and diagonals), the smallest grid.

Tolerances are the evaluation's own: FP64 1e-10 of |F| and 1e-8 of max|df|, FP32 2e-6 and 1e-4."""
import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine, PREC_FP64, PREC_MIXED
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("mmax,dims,box", [(0, (2, 4, 6), (1.0, 2.0, 3.0)), (1, (8, 12, 18), (4.0, 6.0, 9.0)),
                                           (2, (12, 12, 6), (6.0, 6.0, 3.0)), (3, (16, 8, 12), (9.0, 4.0, 6.1)),
                                           (4, (8, 12, 8), (4.0, 6.0, 4.0)), (4, (12, 12, 12), (6.0, 6.0, 6.0)),
                                           (5, (6, 8, 12), (3.0, 4.0, 6.0))])
def test_oz_cells(tmp_path, mmax, dims, box, precision):
    ck = cases.ck_path(tmp_path, mmax, kmax=18.0, dk=0.05)
    o = O.Oracle(dims, box, mmax, ck, SV.kT, SV.n0)
    rng = np.random.default_rng(100 * mmax + dims[0])
    o.set_vext(0.8 * rng.standard_normal(o.shape))
    xi = 1.0 + 0.15 * rng.standard_normal(o.shape)
    f0, df0, t0 = o.energy_grad(xi)
    with Engine(dims, box, mmax, ck, temperature=SV.temperature, n0=SV.n0, precision=precision) as e:
        e.set_vext(o.get_vext())
        f1, df1, t1 = e.energy_and_gradient(xi)
    etol, gtol = (1e-10, 1e-8) if precision == PREC_FP64 else (2e-6, 1e-4)
    assert abs(f1 - f0) <= etol * abs(f0), (f1, f0)
    assert np.all(np.abs(t1 - t0) <= etol * abs(f0)), (t1, t0)
    assert np.abs(df1 - df0).max() <= gtol * np.abs(df0).max()

"""Every FFT length in every position (square planes, lines, columns) and lengths without a
kernel of their own, through an evaluation against the oracle; FP64 to 1e-10 of |F| and 1e-8 of
max|df|, FP32 to 2e-6 and 1e-4 (the evaluation's own bars)."""
import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine, PREC_FP64, PREC_MIXED
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("dims", [(8, 8, 12), (12, 12, 16), (16, 16, 18), (18, 18, 24), (24, 24, 8), (32, 32, 6), (36, 36, 4),
                                  (48, 48, 2), (54, 54, 2), (64, 64, 2), (72, 72, 2), (96, 96, 2), (128, 128, 2),
                                  (8, 12, 36), (12, 8, 54), (16, 18, 72), (18, 16, 96), (24, 6, 128), (36, 4, 32), (54, 2, 48),
                                  (72, 8, 64), (96, 2, 8), (128, 2, 12), (2, 64, 4), (4, 128, 6), (6, 96, 16), (108, 4, 8),
                                  (4, 144, 2), (6, 4, 162)])
def test_fft_lengths(tmp_path, dims, precision):
    box = tuple(0.5 * n for n in dims)
    ck = cases.ck_path(tmp_path, 1, kmax=14.0, dk=0.05)
    o = O.Oracle(dims, box, 1, ck, SV.kT, SV.n0)
    rng = np.random.default_rng(sum(dims))
    o.set_vext(0.8 * rng.standard_normal(o.shape))
    xi = 1.0 + 0.15 * rng.standard_normal(o.shape)
    f0, df0, t0 = o.energy_grad(xi)
    with Engine(dims, box, 1, ck, temperature=SV.temperature, n0=SV.n0, precision=precision) as e:
        e.set_vext(o.get_vext())
        f1, df1, t1 = e.energy_and_gradient(xi)
    etol, gtol = (1e-10, 1e-8) if precision == PREC_FP64 else (2e-6, 1e-4)
    size = max(abs(f0), np.abs(t0).max())
    assert abs(f1 - f0) <= etol * size, (f1, f0)
    assert np.all(np.abs(t1 - t0) <= etol * size), (t1, t0)
    assert np.abs(df1 - df0).max() <= gtol * np.abs(df0).max()

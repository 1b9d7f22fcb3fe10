"""The angular transforms of an FP64 point on the warp-level matrix instructions, against the
oracle where their tiling can go wrong: point counts that leave a remainder in every tile, odd
numbers of orientations, matrices in several column chunks and K slabs, fields at addresses of 8
modulo 16, the excess seam's accumulation, and densities over ten decades (the table logarithm).

Tolerances are the evaluation's own (FP64 1e-10 of |F|, 1e-8 of max|df|; FP32 2e-6, 1e-4).  The
ideal term is held to 1e-12 of its own terms: the table logarithm's 2^-52 max(1, |log x|) and the
sums' rounding stay below 1e-14 of them."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from mdft_b200 import Engine, PREC_FP64, PREC_MIXED
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT
SYSTEMS = [(0, (2, 2, 2)), (1, (6, 6, 6)), (2, (6, 4, 6)), (2, (18, 12, 8)), (3, (6, 6, 6)), (3, (12, 12, 12)),
           (4, (6, 8, 6)), (5, (4, 6, 6)), (5, (12, 8, 8))]


def system(tmp_path, mmax, dims, precision, offset=0):
    box = tuple(0.5 * n for n in dims)
    ck = cases.ck_path(tmp_path, mmax, kmax=14.0, dk=0.05)
    o = O.Oracle(dims, box, mmax, ck, SV.kT, SV.n0)
    rng = np.random.default_rng(7 * mmax + dims[0])
    o.set_vext(3.0 * rng.standard_normal(o.shape))
    xi = np.exp(np.log(10.0) * rng.uniform(-9.5, 0.4, o.shape))
    xi[rng.random(o.shape) < 0.1] = 0.0
    e = Engine(dims, box, mmax, ck, temperature=SV.temperature, n0=SV.n0, precision=precision)
    e.set_vext(o.get_vext())
    return o, e, xi


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("mmax,dims", SYSTEMS)
def test_angular_mma(tmp_path, mmax, dims, precision):
    o, e, xi = system(tmp_path, mmax, dims, precision)
    f0, df0, t0 = o.energy_grad(xi)
    etol, gtol = (1e-10, 1e-8) if precision == PREC_FP64 else (2e-6, 1e-4)
    size, top = max(abs(t0).max(), abs(f0)), np.abs(df0).max()
    buf = torch.zeros(2, xi.size + 1, dtype=torch.float64, device="cuda")
    for off in (0, 1):  # the second time every row starts at 8 modulo 16
        buf[0, off:off + xi.size] = torch.from_numpy(xi.reshape(-1)).cuda()
        torch.cuda.synchronize()
        base = buf.data_ptr()
        step = buf.stride(0) * 8
        f1, t1 = e.energy_and_gradient_device(base + 8 * off, base + step + 8 * (off ^ (buf.stride(0) & 1)))
        df1 = buf[1, off ^ (buf.stride(0) & 1):][:xi.size].cpu().numpy().reshape(xi.shape)
        assert abs(f1 - f0) <= etol * size, (off, f1, f0)
        assert np.all(np.abs(t1 - t0) <= etol * size), (off, t1, t0)
        assert np.abs(df1 - df0).max() <= gtol * top, off
        f2, t2 = e.energy_and_gradient_device(base + 8 * off, None)
        assert f2 == f1 and np.array_equal(t1, t2)
    if precision == PREC_FP64:
        rho, w = xi ** 2 * e.rho0, e.weights
        lg = np.log(np.where(rho > 0, xi ** 2, 1.0))
        each = np.where(rho > np.finfo(float).eps, rho * lg - rho + e.rho0, e.rho0) * w * e.dv * e.kT
        assert abs(t1[0] - each.sum()) <= 1e-12 * np.abs(each).sum()
    acc = np.full(xi.shape, 0.25)
    fexc = e.excess_energy(xi, acc)
    dfid = np.where(rho > np.finfo(float).eps, w * 2 * e.rho0 * xi * (SV.kT * lg + o.get_vext()), 0.0) if precision == PREC_FP64 else None
    assert abs(fexc - t0[2]) <= etol * size
    if dfid is not None:
        assert np.abs(acc - 0.25 - (df0 - dfid)).max() <= gtol * top
    e.close()

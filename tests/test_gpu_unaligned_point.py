"""Evaluations of a device point at an address of 8 modulo 16 on grids whose CTAs walk many tiles,
every stage of the projection's ring filled several times: the same evaluation as at an aligned
address, against the oracle at the FP64 and mixed bars (F 1e-10 / 2e-6, gradient 1e-8 / 1e-4)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from mdft_b200 import Engine, PREC_FP64, PREC_MIXED, synth
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("mmax,mrso,dims", [(1, 2, (96, 96, 64)), (1, 3, (96, 96, 64)), (2, 2, (48, 48, 32)), (0, 2, (96, 96, 64))])
def test_unaligned_point(tmp_path, mmax, mrso, dims, precision):
    box = tuple(0.5 * n for n in dims)
    ck = synth.make_ck_file(str(tmp_path / "ck.txt"), mmax, mrso=mrso, kmax=12.0, dk=0.05)
    e = Engine(dims, box, mmax, ck, temperature=SV.temperature, n0=SV.n0, mrso=mrso, precision=precision)
    rng = np.random.default_rng(mmax + 10 * mrso)
    e.set_vext(0.8 * rng.standard_normal(e.shape))
    xi = 1.0 + 0.15 * rng.standard_normal(e.shape)
    n = xi.size
    res = []
    for off in (0, 1):
        x, g = (torch.zeros(n + 2, dtype=torch.float64, device="cuda") for _ in range(2))
        x[off:off + n] = torch.from_numpy(xi.reshape(-1)).cuda()
        torch.cuda.synchronize()
        f, t = e.energy_and_gradient_device(x.data_ptr() + 8 * off, g.data_ptr() + 8 * off)
        torch.cuda.synchronize()
        res.append((f, t, g[off:off + n].cpu().numpy().reshape(xi.shape)))
    etol, gtol = (1e-10, 1e-8) if precision == PREC_FP64 else (2e-6, 1e-4)
    (f0, t0, g0), (f1, t1, g1) = res
    assert abs(f1 - f0) <= etol * abs(f0) and np.all(np.abs(t1 - t0) <= etol * abs(f0)), (f0, f1)
    assert np.abs(g1 - g0).max() <= gtol * np.abs(g0).max()
    o = O.Oracle(dims, box, mmax, ck, SV.kT, SV.n0, mrso=mrso)
    o.set_vext(e.get_vext())
    fo, go, to = o.energy_grad(xi)
    assert abs(f1 - fo) <= etol * abs(fo) and np.all(np.abs(t1 - to) <= etol * abs(fo)), (f1, fo)
    assert np.abs(g1 - go).max() <= gtol * np.abs(go).max()
    e.close()

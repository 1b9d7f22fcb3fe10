"""A hard-sphere bridge's error is reported once, by the call that ran the bridge: the excess term
alone (which runs none) is evaluated as on a handle without one, before any full evaluation, after
a failed one, after a failed energy_bridge, and after the bridge was set again."""
import numpy as np
import pytest

from oracle import oracle as O
from mdft_b200 import Engine, MdftError
import cases

pytestmark = pytest.mark.gpu
SV = cases.SOLVENT


@pytest.mark.parametrize("functional", [1, 2])
def test_excess_energy_beside_a_failed_bridge(tmp_path, functional):
    c = cases.ALL_CASES["mol16_m2"]
    ck = cases.case_ck(tmp_path, c)
    o = O.Oracle(c["n"], c["L"], c["mmax"], ck, SV.kT, SV.n0)
    xi = cases.xi_of(c, o.shape, amp=0.3)
    dense = 3.0 * np.ones(o.shape)  # n3 >= 1
    f0, _, t0 = o.energy_grad(xi)
    with Engine(c["n"], c["L"], c["mmax"], ck, temperature=SV.temperature, n0=SV.n0) as e:
        e.set_bridge_fmt(functional, 1.4)

        def excess():
            assert abs(e.excess_energy(xi) - t0[2]) <= 1e-10 * abs(f0)

        excess()  # the handle's first call
        with pytest.raises(MdftError, match="hard-sphere"):
            e.energy_and_gradient(dense)
        excess()
        excess()
        with pytest.raises(MdftError, match="hard-sphere"):
            e.bridge_energy(dense)
        excess()
        with pytest.raises(MdftError, match="hard-sphere"):  # still an error wherever the bridge runs
            e.energy_and_gradient(dense)
        e.set_bridge_fmt(functional, 1.4)
        excess()
        f, _, _ = e.energy_and_gradient(xi)
        assert np.isfinite(f)

"""The one-launch projection (up to 160 orbitals) and the stepwise one past it
against the eigensolver route, at tile edges of the projection (orbital counts
around multiples of 8, the smallest and the largest it takes) and with one
occupied orbital. Both routes converge the same float64 SCF to |dE| < 1e-8 and
a commutator below 1e-6, whose square bounds the energies' difference: 1e-10 Ha
as in test_gpu_purify.py."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,charges", [("water", None), ("alkane1", None), ("water2", None),
                                          ("alkane2", None), ("water5", None), ("water6", None),
                                          ("water", (1.0, 0.5, 0.5))])
def test_projection_sizes(name, charges):
    from dftax_b200 import df, systems
    from dftax_b200.ks import KS, scf

    sym, xyz, orb, aux, _ = systems.workload(name, seed=6)
    e = {}
    for density in ("eigh", "purify"):
        ks = KS(sym, xyz, orb, coulomb=df(aux), xc="HF", charges=charges, density=density)
        r = scf(ks)
        assert r.converged
        e[density] = r
        # (the guess goes to the eigensolver; an iteration without a gap may)
        assert r.n_eig <= (2 if density == "purify" else r.n_iter + 1), (density, r.n_eig, r.n_iter)
    assert abs(e["eigh"].e_tot - e["purify"].e_tot) < 1e-10
    assert np.abs(e["eigh"].P - e["purify"].P).max() < 1e-5
    assert np.abs(e["eigh"].mo_energy - e["purify"].mo_energy).max() < 1e-5

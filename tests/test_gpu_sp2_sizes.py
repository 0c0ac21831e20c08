"""The one-launch projection (up to 160 orbitals) and the stepwise one past it
against the eigensolver route: 30 to 180 orbitals of the named sets, one occupied
orbital, and sets made for the tile edges: 8, 16 and 48 orbitals (whole tiles of
8), 152 and 160 (the last tile row and the largest it takes: 210 tiles, four a
warp), 153 (one orbital in the last tile row) and 161 (the first stepwise one).
Both routes converge the same float64 SCF to |dE| < 1e-8 and a commutator below
1e-6, whose square bounds the energies' difference: 1e-10 Ha as in
test_gpu_purify.py."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,charges", [("water", None), ("alkane1", None), ("water2", None),
                                          ("alkane2", None), ("water5", None), ("water6", None),
                                          ("water", (1.0, 0.5, 0.5))])
def test_projection_sizes(name, charges):
    from dftax_b200 import systems

    compare(*systems.workload(name, seed=6)[:4], charges)


def compare(sym, xyz, orb, aux, charges=None):
    from dftax_b200 import df
    from dftax_b200.ks import KS, scf

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
    return e["purify"]


# contracted core, then valence exponents in turn
O_S = [(0, [130.7, 23.8, 6.44], [0.154, 0.535, 0.444]), (0, [2.0], [1.0]), (0, [0.7], [1.0]),
       (0, [0.25], [1.0])]
O_P = [(1, [5.0, 1.2], [0.4, 0.7]), (1, [0.4], [1.0])]
O_D = [(2, [0.9], [1.0])]
H_S = [(0, [3.4, 0.62], [0.3, 0.8]), (0, [0.17], [1.0])]
H_P = [(1, [0.8], [1.0])]


@pytest.mark.parametrize("n,o,h,nmo", [(1, (3, 1, 0), (1, 0), 8), (1, (3, 1, 0), (2, 1), 16),
                                       (3, (3, 1, 0), (2, 1), 48), (8, (3, 2, 0), (2, 1), 152),
                                       (9, (4, 1, 0), (2, 1), 153), (8, (4, 2, 0), (2, 1), 160),
                                       (7, (2, 2, 1), (2, 1), 161)])
def test_projection_at_tile_edges(n, o, h, nmo):
    from dftax_b200 import build_basis_data, systems

    sym, xyz = systems.water_cluster(n, seed=6)
    orb = build_basis_data(sym, xyz, {"O": O_S[:o[0]] + O_P[:o[1]] + O_D[:o[2]],
                                      "H": H_S[:h[0]] + H_P[:h[1]]})
    r = compare(sym, xyz, orb, systems.basis_for(sym, xyz)[1])
    assert r.mo_energy.shape[-1] == nmo

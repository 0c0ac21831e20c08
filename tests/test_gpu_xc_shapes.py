"""XC energy and matrix at the sizes where the quadrature kernels' tiles end:
point counts around the 64-point blocks and 512-point slices, chunks of 256 to
8192 points, 30 to 114 functions (one and two 64-column blocks, even and odd
counts), with and without the matrix, against the oracle's dense quadrature.

Tolerance: sums of up to 5000 x 114^2 float64 products, 2^-53 * sqrt of that
< 1e-12 relative.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-12


@pytest.mark.parametrize("name,npts,chunk", [("water", 1, 256), ("water", 63, 256), ("water", 65, 512),
                                             ("water3", 1000, 256), ("water3", 4097, 768),
                                             ("alkane1", 5000, 8192), ("alkane2", 2500, 2048)])
def test_xc_shapes(name, npts, chunk):
    import torch

    from dftax_b200 import df, systems
    from dftax_b200.ks import KS
    from oracle import ks as oks

    sym, xyz, orb, aux, nocc = systems.workload(name, seed=1)
    rng = np.random.default_rng(npts)
    pts = xyz[rng.integers(0, len(xyz), npts)] + rng.standard_normal((npts, 3))
    w = rng.uniform(0.01, 0.1, npts)
    ks = KS(sym, xyz, orb, coulomb=df(aux), grid=(pts, w), grid_chunk=chunk)
    C = systems.random_occupied(orb.nao, nocc, seed=3)
    P = 2.0 * C @ C.T
    e0, V0 = oks.exc_and_vxc(orb, pts, w, P)
    for _ in range(3):   # direct, captured, replayed; the caller's buffers change
        e, V = ks.xc_energy(torch.as_tensor(P, device="cuda"))
        assert abs(e - e0) <= REL * abs(e0)
        assert np.linalg.norm(V.cpu().numpy() - V0) <= REL * np.linalg.norm(V0)
    e1, none = ks.xc_energy(P, want_fock=False)
    assert none is None and abs(e1 - e0) <= REL * abs(e0)


@pytest.mark.parametrize("npts,far", [(2047, 30.0), (2049, 300.0), (6000, 1e5), (5000, 1e7)])
def test_scattered_points(npts, far):
    """The device sort of the grid at tile edges (2048 points), with many points in
    one cell (equal keys) and with one to eight digits of key: half of the points
    lie up to `far` Bohr out, where the density vanishes."""
    import torch

    from dftax_b200 import df, systems
    from dftax_b200.ks import KS
    from oracle import ks as oks

    sym, xyz, orb, aux, nocc = systems.workload("water", seed=1)
    rng = np.random.default_rng(npts)
    pts = xyz[rng.integers(0, len(xyz), npts)] + rng.standard_normal((npts, 3))
    pts[::2] += rng.uniform(-far, far, pts[::2].shape)
    w = rng.uniform(0.01, 0.1, npts)
    C = systems.random_occupied(orb.nao, nocc, seed=3)
    P = 2.0 * C @ C.T
    e0, V0 = oks.exc_and_vxc(orb, pts, w, P)
    e = []
    for _ in range(2):
        ks = KS(sym, xyz, orb, coulomb=df(aux), grid=(pts, w), grid_chunk=512)
        e1, V = ks.xc_energy(torch.as_tensor(P, device="cuda"))
        assert abs(e1 - e0) <= REL * abs(e0)
        assert np.linalg.norm(V.cpu().numpy() - V0) <= REL * np.linalg.norm(V0)
        e.append(e1)
        ks.close()
    assert e[0] == e[1]


def test_many_chunks_without_functions():
    """More chunks that no function reaches than a launch dimension holds (65535):
    16.8 million far points beside 4096 near ones, 256 points a chunk. They add
    nothing: the result is that of the near points alone."""
    import torch

    from dftax_b200 import df, systems
    from dftax_b200.ks import KS

    sym, xyz, orb, aux, nocc = systems.workload("water", seed=1)
    rng = np.random.default_rng(0)
    near = xyz[rng.integers(0, len(xyz), 4096)] + rng.standard_normal((4096, 3))
    w = rng.uniform(0.01, 0.1, 4096)
    far = 65540 * 256
    pts = np.full((far + 4096, 3), 300.0)
    pts[far // 2:far // 2 + 4096] = near
    ws = np.full(far + 4096, 0.5)
    ws[far // 2:far // 2 + 4096] = w
    C = systems.random_occupied(orb.nao, nocc, seed=3)
    P = torch.as_tensor(2.0 * C @ C.T, device="cuda")
    out = []
    for grid in ((near, w), (pts, ws)):
        ks = KS(sym, xyz, orb, coulomb=df(aux), grid=grid, grid_chunk=256)
        for _ in range(3):   # direct, captured, replayed
            e, V = ks.xc_energy(P)
        out.append((e, V))
        ks.close()
    (e0, V0), (e1, V1) = out
    assert abs(e1 - e0) <= REL * abs(e0)
    assert float((V1 - V0).norm()) <= REL * float(V0.norm())


def test_no_chunk_has_functions():
    """A grid that no function reaches: zero energy and matrix."""
    import torch

    from dftax_b200 import df, systems
    from dftax_b200.ks import KS

    sym, xyz, orb, aux, nocc = systems.workload("water", seed=1)
    ks = KS(sym, xyz, orb, coulomb=df(aux), grid=(np.full((700, 3), 300.0), np.ones(700)),
            grid_chunk=256)
    C = systems.random_occupied(orb.nao, nocc, seed=3)
    for _ in range(3):
        e, V = ks.xc_energy(torch.as_tensor(2.0 * C @ C.T, device="cuda"))
        assert e == 0.0 and not V.any()


def test_chunk_larger_than_a_launch():
    """A chunk size whose 512-point slices exceed a launch dimension is cut: H2 with
    an s shell on each atom, as with ordinary chunks."""
    import torch

    from dftax_b200 import build_basis_data, df
    from dftax_b200.ks import KS

    xyz = np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]])
    orb = build_basis_data(["H", "H"], xyz, {"H": [(0, [0.8], [1.0])]})
    aux = build_basis_data(["H", "H"], xyz, {"H": [(0, [1.1], [1.0])]})
    rng = np.random.default_rng(4)
    grid = (xyz[rng.integers(0, 2, 3000)] + rng.standard_normal((3000, 3)), rng.uniform(0.01, 0.1, 3000))
    P = torch.tensor([[0.6, 0.5], [0.5, 0.6]], dtype=torch.float64, device="cuda")
    out = []
    for chunk in (256, 1 << 26):
        ks = KS(["H", "H"], xyz, orb, coulomb=df(aux), grid=grid, grid_chunk=chunk)
        out.append(ks.xc_energy(P))
        ks.close()
    (e0, V0), (e1, V1) = out
    assert abs(e1 - e0) <= REL * abs(e0)
    assert float((V1 - V0).norm()) <= REL * float(V0.norm())

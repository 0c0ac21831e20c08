"""J and K of float64 and mixed plans at the sizes where the contraction
kernels' tiles end: every column tile of the half transform (8 to 80, one and
several tiles, odd counts), one and several 64-row tiles of K, k slices that do
not divide, screened pairs, signed weights. The reference is the plan's own
dense (mn|P) and V+ contracted in float64 by torch.

Float64 tolerance: the two sides round (mn|P) V+ (ls|Q) in different orders,
which the metric's condition number (<= 1e7 kept) amplifies: 1e7 * 2^-53 *
sqrt(naux) < 5e-8 at worst, 5e-10 seen across the repository's parity tests.
Mixed tolerance: the digits' 2^-32 of each row's scale, amplified the same way
in B only: 1e-8 for J, 1e-7 for K (tests/test_gpu_mixed.py).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a - b).norm() / b.norm())


def dense_jk(plan, C, w):
    import torch

    T, V = plan.eri3c_dense(), plan.metric_pinv()
    D = (C * w) @ C.T
    J = T @ (V @ torch.einsum("mnP,mn->P", T, D))
    X = torch.einsum("mnP,ni->miP", T, C)
    K = torch.einsum("miP,PQ,niQ->mn", X * w[None, :, None], V, X)
    return J, K


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name,screen,ncols", [
    ("water", None, (1, 5, 8, 9, 17, 30)),
    ("water3", None, (24, 25, 40, 41, 64, 81, 90)),
    ("alkane4", 1e-8, (16, 33, 57, 97)),
])
def test_jk_shapes(name, screen, ncols, precision):
    import torch

    from dftax_b200 import Plan, systems

    sym, xyz, orb, aux, _ = systems.workload(name, seed=5)
    plan = Plan(orb, aux, screen=screen, precision=precision).build()
    tj, tk = (5e-10, 5e-10) if precision == "fp64" else (1e-8, 1e-7)
    for ncol in ncols:
        C = torch.as_tensor(systems.random_occupied(plan.nao, ncol, seed=ncol), device="cuda")
        w = torch.ones(ncol, dtype=torch.float64, device="cuda")
        J, K = plan.jk(C)
        Jr, Kr = dense_jk(plan, C, w)
        assert rel(J, Jr) < tj and rel(K, Kr) < tk, (ncol, rel(J, Jr), rel(K, Kr))
        assert torch.equal(K, K.T)
        J2, K2 = plan.jk(C)
        assert torch.equal(J, J2) and torch.equal(K, K2)
        if ncol > 2:   # signed weights: columns gathered in two passes
            w = torch.linspace(1.5, -1.0, ncol, dtype=torch.float64, device="cuda")
            J, K = plan.jk(C, w)
            Jr, Kr = dense_jk(plan, C, w)
            # the rounding is relative to the sum without cancellation
            Ja, Ka = dense_jk(plan, C, w.abs())
            assert float((J - Jr).norm() / Ja.norm()) < tj, ncol
            assert float((K - Kr).norm() / Ka.norm()) < tk, ncol
    assert np.isfinite(float(K.sum()))

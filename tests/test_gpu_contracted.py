"""Contracted shells with unequal primitive counts (1, 2 and 3 within one
angular momentum) through the integral kernels that give a group of lanes to a
shell pair or triple: metric, 3-center rows and the gradient, against the
compiled CPU oracle. Shell counts leave the lane groups partly filled.

Tolerances: integrals 1e-12 absolute on values of order one (sums of up to 27
primitive triples of 1e-14 each); the gradient as in test_gpu_grad.py, 1e-9 of
the largest component for pure Coulomb with the device's own V+.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORB = {"O": [(0, [6.0, 1.5, 0.4], [0.3, 0.5, 0.4]), (0, [0.25], [1.0]), (1, [2.0, 0.5], [0.6, 0.6]),
             (1, [0.3], [1.0]), (2, [1.0, 0.4], [0.5, 0.7])],
       "H": [(0, [2.0, 0.5], [0.4, 0.8]), (0, [0.2], [1.0]), (1, [0.8], [1.0])]}
AUX = {"O": [(0, [8.0, 2.0], [0.5, 0.5]), (0, [0.9], [1.0]), (0, [0.3], [1.0]),
             (1, [1.5, 0.6, 0.25], [0.3, 0.5, 0.3]), (2, [1.2], [1.0]), (2, [0.9, 0.4], [0.6, 0.6]),
             (3, [1.0, 0.5], [0.7, 0.4])],
       "H": [(0, [1.0], [1.0]), (0, [0.4, 0.15], [0.5, 0.5]), (1, [0.7], [1.0]), (2, [0.8], [1.0])]}


def _bases(n):
    from dftax_b200 import build_basis_data, systems

    sym, xyz = systems.water_cluster(n, seed=2)
    return xyz, build_basis_data(sym, xyz, ORB), build_basis_data(sym, xyz, AUX)


@pytest.mark.parametrize("n", [1, 2])
def test_integrals(n):
    from dftax_b200 import Plan
    from oracle import cpu

    _, orb, aux = _bases(n)
    plan = Plan(orb, aux)
    V = plan.eri2c_dense().cpu().numpy()
    assert np.abs(V - cpu.eri2c(aux)).max() < 1e-12 * max(1.0, np.abs(V).max())
    assert np.array_equal(V, V.T)
    T = plan.eri3c_dense().cpu().numpy()
    assert np.abs(T - cpu.eri3c_dense(orb, aux)).max() < 1e-12 * max(1.0, np.abs(T).max())


@pytest.mark.parametrize("n,hf", [(1, 0.0), (2, 0.0), (1, 0.25)])
def test_gradient(n, hf):
    from dftax_b200 import Plan, systems
    from oracle import cpu

    xyz, orb, aux = _bases(n)
    C = systems.random_occupied(orb.nao, 5 * n, seed=n)
    P = 2.0 * C @ C.T
    plan = Plan(orb, aux).build()
    _, g = plan.energy_grad(P, hf, xyz)
    _, ref = cpu.df_energy_grad(orb, aux, P, hf, xyz, vinv=plan.metric_pinv().cpu().numpy())
    tol = 1e-9 if hf == 0.0 else 5e-8
    assert np.abs(g - ref).max() <= tol * max(1.0, np.abs(ref).max())

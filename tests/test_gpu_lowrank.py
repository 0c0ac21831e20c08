"""Energy and Fock of densities through the pivoted Cholesky factor and through
the eigensolver it falls back to: every rank from zero to full, one and two
channels, graded eigenvalues down to the cutoff, an indefinite and a negative
density. The reference contracts the plan's own dense (mn|P) and V+ in float64.

Tolerance: rounding of (mn|P) V+ amplified by the metric's condition number,
5e-10 (see test_gpu_jk_shapes.py), relative to |J| + |K| of the density without
cancellation; a factor accepted with a residual of 3e-14 max |P| per element
moves K by less than nao * 3e-14 of that, below it.
"""

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 5e-10


def _densities(n, rng):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    occ = lambda r: 2.0 * q[:, :r] @ q[:, :r].T  # noqa: E731
    graded = (q * 10.0 ** -np.linspace(0.0, 16.0, n)) @ q.T
    yield "rank 1", occ(1)[None]
    yield "rank n/3", occ(n // 3)[None]
    yield "full rank", occ(n)[None]
    yield "zero", np.zeros((1, n, n))
    yield "graded", 0.5 * (graded + graded.T)[None]
    yield "open shell, one empty channel", np.stack([0.5 * occ(n // 3), np.zeros((n, n))])
    yield "open shell", np.stack([0.5 * occ(7), 0.5 * occ(5)])
    yield "indefinite", (occ(5) - 0.3 * occ(9))[None]
    yield "zero diagonal", np.kron(np.eye(n // 2), [[0.0, 1.0], [1.0, 0.0]])[None]
    yield "negative", -occ(4)[None]


@pytest.mark.parametrize("name,precision,hf_lr", [("water", "fp64", 0.0), ("alkane2", "fp64", 0.0),
                                                  ("water3", "mixed", 0.0), ("water", "fp64", 0.4)])
def test_energy_of_any_density(name, precision, hf_lr):
    import torch

    from dftax_b200 import Plan, systems

    sym, xyz, orb, aux, _ = systems.workload(name, seed=3)
    plan = Plan(orb, aux, precision=precision, omega=0.3 if hf_lr else 0.0).build()
    terms = [(plan, 0.25)] + ([(plan.long_range, hf_lr)] if hf_lr else [])
    T, V = plan.eri3c_dense(), plan.metric_pinv()
    rel = REL if precision == "fp64" else 1e-7
    for what, P in _densities(orb.nao, np.random.default_rng(1)):
        Pt = torch.as_tensor(P, device="cuda")
        e, F = plan.energy(Pt, 0.25, hf_coeff_lr=hf_lr)
        g = torch.einsum("mnP,mn->P", T, Pt.sum(0))
        J = T @ (V @ g)
        ref, size = 0.5 * float(g @ (V @ g)), float(J.norm())
        Fr = J[None].repeat(len(P), 1, 1)
        half = 0.5 if len(P) == 1 else 1.0
        for p, a in terms:
            t, v = (T, V) if p is plan else (p.eri3c_dense(), p.metric_pinv())
            for s in range(len(P)):
                Y = torch.einsum("mlP,ls->msP", t, Pt[s])
                K = torch.einsum("msP,PQ,nsQ->mn", Y, v, t)
                ref -= 0.5 * half * a * float((Pt[s] * K).sum())
                Fr[s] -= half * a * K
                A = torch.linalg.eigh(Pt[s])
                A = (A[1] * A[0].abs()) @ A[1].T
                size += float(torch.einsum("mlP,ls,PQ,nsQ->mn", t, A, v, t).norm())
        assert float((F - Fr).norm()) <= rel * size, (what, float((F - Fr).norm()), size)
        assert abs(e - ref) <= rel * size * max(float(Pt.norm()), 1e-300), (what, e, ref)
        e2, F2 = plan.energy(Pt, 0.25, hf_coeff_lr=hf_lr)
        assert e2 == e and torch.equal(F, F2), what


def test_sizes_on_two_threads():
    """Threads that factor densities of different sizes at once, each on its own
    context and stream: every energy is the one of a lone call."""
    import threading

    import torch

    from dftax_b200 import Plan, systems
    from dftax_b200.coulomb import Context

    plans, dens, alone = [], [], []
    for name in ("water", "water6"):
        _, _, orb, aux, nocc = systems.workload(name, seed=2)
        plans.append(Plan(orb, aux, ctx=Context(0)).build())
        C = systems.random_occupied(orb.nao, nocc, seed=5)
        dens.append(torch.as_tensor(2.0 * C @ C.T, device="cuda"))
        alone.append(plans[-1].energy(dens[-1], 0.25)[0])
    errors = []

    def work(q):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    assert abs(plans[q].energy(dens[q], 0.25)[0] - alone[q]) <= 1e-10 * abs(alone[q])
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(q,)) for q in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_mixed_factor_is_as_precise_as_eigenvectors():
    """K of an occupied density through the factor of a mixed plan is no further
    from the float64 plan's K than through the density's eigenvectors. The digits
    of a column are relative to its largest element, so the columns' shape sets the
    error; over twelve molecules of 10 to 30 columns the two sides' independent
    roundings give errors of about the same size (ratio 0.88 here; the bare Cholesky
    columns fail). The bound is a tenth above equality."""
    import torch

    from dftax_b200 import Plan, systems

    factor = eig = 0.0
    for name, seed in itertools.product(("water3", "alkane2", "alkane4", "water6"), range(3)):
        sym, xyz, orb, aux, nocc = systems.workload(name, seed=seed)
        exact, mixed = (Plan(orb, aux, precision=p).build() for p in ("fp64", "mixed"))
        C = torch.as_tensor(systems.random_occupied(orb.nao, nocc, seed=seed), device="cuda")
        P = C @ C.T
        w, U = torch.linalg.eigh(P)
        U = (U[:, -nocc:] * w[-nocc:].sqrt()).contiguous()
        K0 = exact.jk(C, want_j=False)[1]
        _, F = mixed.energy(P[None], 2.0)    # F = J - K
        J, K = mixed.jk(U)
        F = F.reshape(J.shape)
        factor += float(((J - F - K0).norm() / K0.norm()) ** 2)
        eig += float(((K - K0).norm() / K0.norm()) ** 2)
    print("factor / eigenvectors:", (factor / eig) ** 0.5)
    assert factor <= 1.1 ** 2 * eig, (factor / eig) ** 0.5


@pytest.mark.parametrize("n", [6, 35])
def test_rank_cap(n):
    """Ranks at the columns where the factor gives way: the gradient's half of the
    functions, Fock's half past 1024 functions (35 waters: 1050), full rank, and
    densities whose residual turns negative at once, after some columns and after
    nearly all. One s shell on each oxygen as the auxiliary set keeps the
    contractions small."""
    import torch

    from dftax_b200 import Plan, build_basis_data, systems

    sym, xyz = systems.water_cluster(n, seed=1)
    orb, _ = systems.basis_for(sym, xyz)
    ox = [i for i, s in enumerate(sym) if s == "O"]
    aux = build_basis_data(["O"] * n, xyz[ox], {"O": [(0, [0.8], [1.0])]})
    plan = Plan(orb, aux).build()
    T, V = plan.eri3c_dense(), plan.metric_pinv()
    m = orb.nao
    g = torch.Generator().manual_seed(n)
    q = torch.linalg.qr(torch.randn(m, m, generator=g, dtype=torch.float64).cuda())[0]
    w = torch.rand(m, generator=g, dtype=torch.float64).cuda() + 0.1

    def form(q, w):
        P = (q * w) @ q.T
        return 0.5 * (P + P.T)

    half = m // 2
    cases = [form(q[:, :r], w[:r]) for r in (half - 1, half, half + 1, m)]
    cases += [form(q, w - 0.12), form(q[:, :20], torch.sign(w[:20] - 0.6)),
              form(q[:, :half], torch.where(torch.arange(half, device="cuda") < half - 2, 1.0, -1e-3))]
    for P in cases:
        J = T @ (V @ torch.einsum("mnP,mn->P", T, P))
        X = torch.einsum("mnP,PQ->mnQ", T, torch.linalg.cholesky(V))
        K = torch.einsum("mlQ,ls,nsQ->mn", X, P, X)
        F0 = J - 0.125 * K
        e0 = 0.5 * float((J * P).sum()) - 0.0625 * float((K * P).sum())
        e, F = plan.energy(P[None], 0.25)
        assert float((F.reshape(F0.shape) - F0).norm()) < REL * float(J.norm() + K.norm())
        assert abs(e - e0) < REL * float((J * P).abs().sum() + (K * P).abs().sum())
        if n == 6:   # both forms of the gradient's K part: the energy goes through it
            eg, _ = plan.energy_grad(P[None], 0.25, xyz)
            assert abs(eg - e0) < REL * float((J * P).abs().sum() + (K * P).abs().sum())

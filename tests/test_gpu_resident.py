"""Resident form (one CTA per trajectory) at the edges of its launch shapes, against the oracle.

The launch shape changes at D = 32, 64, 128, 256 and 512, a thread keeps 16 entries of a row of H
in registers, and the small exponential changes from its Taylor series to the Pade form at a large
norm.  complex128: per-trajectory yields within 1e-10 relative of the oracle (modified Gram-Schmidt
Arnoldi, Pade); complex64: 1e-6, the precision form's target.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from oracle import density as den
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _run(H, system, F, times, m, precision, kappa=None, K=None, form="resident", recurrence=L.REC_AUTO, budget=0):
    with hs.HSPropagatorB200(0, budget) as p:
        p.set_form(form)
        p.set_hamiltonian(*H)
        p.set_reaction(kappa=kappa, csr=K)
        p.set_electron_pair(*system.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in system.observables()])
        p.set_factors(F)
        p.propagate(times, m, precision, recurrence=recurrence)
        return p.yields()[0]


def _unequal(system):
    system.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
    return sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), system) for k, r in system.sinks.items())


# D = 12, 32, 36, 64, 96, 128, 144, 256, 288, 512, 576 on both sides of every shape's limit
@pytest.mark.parametrize("nuc", [[3], [2] * 3, [3, 3], [2] * 4, [3, 2, 2, 2], [2] * 5, [3, 3, 2, 2], [2] * 6,
                                 [3, 3, 2, 2, 2], [2] * 7, [3, 3, 2, 2, 2, 2]])
@pytest.mark.parametrize("m", [1, 7, 16])
def test_shapes_against_the_oracle(nuc, m):
    s = h.random_system(nuc[::2], nuc[1::2], seed=7 + len(nuc))
    F = s.trace_samples(3, 5.0)
    times = S.time_grid(4.0, 1.0)
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=s.kappa(), krylov=m, nthreads=8)
    H = s.hamiltonian_csr()
    for prec, rec, tol in (("c128", L.REC_AUTO, 1e-10), ("c128", L.REC_ARNOLDI, 1e-10), ("c64", L.REC_AUTO, 1e-6)):
        assert _rel(_run(H, s, F, times, m, prec, s.kappa(), recurrence=rec), ref["traj_yield"]) < tol, (prec, rec)
    K = _unequal(s)
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), K_csr=den.to_csr(K), krylov=m, nthreads=8)
    assert _rel(_run(H, s, F, times, m, "c128", K=den.to_csr(K)), ref["traj_yield"]) < 1e-10


@pytest.mark.parametrize("m", [31, 32])
@pytest.mark.parametrize("dt", [1.0, 4e3])
def test_largest_krylov_dimension_and_long_steps(m, dt):
    # dt = 4000 ns: dt |H| of several hundred takes the Pade form of the small exponential
    s = h.random_system([2, 2], [3], seed=11)
    F = s.trace_samples(3, 5.0)
    times = S.time_grid(dt, dt)
    H, kappa = s.hamiltonian_csr(), 1e-5
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), kappa=kappa, krylov=m, nthreads=8)
    # both sides exponentiate a Krylov matrix of norm dt |H|: rounding grows with it
    tol = 1e-10 * max(1.0, dt / 100)
    for rec in (L.REC_AUTO, L.REC_ARNOLDI):
        assert _rel(_run(H, s, F, times, m, "c128", kappa, recurrence=rec), ref["traj_yield"]) < tol, rec


@pytest.mark.parametrize("hermitian", [True, False])
def test_full_rows_and_a_hamiltonian_that_is_not_hermitian(hermitian):
    """Rows longer than the register part; without H = H^dagger the recurrence has to stay Arnoldi."""
    s = h.random_system([2, 2], [2], seed=12)
    D = s.dim
    rng = np.random.default_rng(3)
    A = 0.03 * (rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    A = 0.5 * (A + A.conj().T) if hermitian else A
    H = den.to_csr(A)
    F = s.trace_samples(4, 6.0)
    times = S.time_grid(3.0, 1.0)
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), kappa=1e-3, krylov=16, nthreads=8)
    assert _rel(_run(H, s, F, times, 16, "c128", 1e-3), ref["traj_yield"]) < 1e-10


def test_one_long_row_and_a_tight_budget_walk_the_csr_rows():
    s = h.random_system([2] * 4, [2] * 3, seed=13)
    D = s.dim
    A = den.dense_hamiltonian(s)
    A[5, :] += 1e-3
    A[:, 5] += 1e-3  # a full row: no padded copy
    F = s.trace_samples(5, 6.0)
    times = S.time_grid(3.0, 1.0)
    H = den.to_csr(A)
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), kappa=s.kappa(), krylov=12, nthreads=8)
    assert _rel(_run(H, s, F, times, 12, "c128", s.kappa()), ref["traj_yield"]) < 1e-10
    assert _rel(_run(H, s, F, times, 12, "c64", s.kappa()), ref["traj_yield"]) < 1e-6
    # the budget ends 2 KB above what the run holds without the copy of H
    H = s.hamiltonian_csr()
    nnz, M = int(H[0][-1]), 5
    need = 4 * (D + 1) + 28 * nnz + 16 * D * 64 + 16 * D * M + 3 * 4 * 8 * 64 + 8 * 4 * 4 * M + 8 * 16 * 16 + 2048
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), kappa=s.kappa(), krylov=12, nthreads=8)
    assert _rel(_run(H, s, F, times, 12, "c128", s.kappa(), budget=need), ref["traj_yield"]) < 1e-10


@pytest.mark.parametrize("D,M,full", [(64, 5, True), (12, 1, False), (576, 2, False)])
def test_noalloc_step_on_full_rows_and_uneven_shapes(D, M, full):
    import torch
    rng = np.random.default_rng(D)
    if full:
        A = 0.03 * (rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
        H = den.to_csr(0.5 * (A + A.conj().T))
    else:
        H = h.random_system([3] if D == 12 else [3, 3, 2, 2, 2, 2], [], seed=14).hamiltonian_csr()
    psi = rng.normal(size=(M, D)) + 1j * rng.normal(size=(M, D))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (*H, psi)]
    out = torch.empty_like(dev[3])
    rc = L.lib.msgpu_krylov_step_noalloc(D, *(t.data_ptr() for t in dev[:3]), 2e-3, M, dev[3].data_ptr(),
                                         out.data_ptr(), 1.0, min(12, D), torch.cuda.current_stream().cuda_stream)
    assert rc == L.MSGPU_OK
    ref = np.stack([orc.krylov_expm(H, 2e-3, b, 1.0, min(12, D)) for b in psi])
    assert np.max(np.abs(out.cpu().numpy() - ref)) / np.max(np.abs(ref)) < 1e-12

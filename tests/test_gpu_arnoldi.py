"""Arnoldi forms with a second Gram-Schmidt pass and at every accumulator batch, against the oracle.

H = c I + a radical pair's H makes G v nearly parallel to v, so that orthogonalisation cancels
most of it and the second pass runs.  complex128 within 1e-10 of the oracle's modified
Gram-Schmidt; complex64 within 1e-6 (its U = H v carries FP32 rounding of c).
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


def _run(H, s, F, times, m, precision, form, K):
    with hs.HSPropagatorB200(0) as p:
        p.set_form(form)
        p.set_hamiltonian(*H)
        p.set_reaction(csr=K)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(times, m, precision)
        return p.yields()[0]


def _case(nuc, seed, shift):
    s = h.random_system(nuc[::2], nuc[1::2], seed=seed)
    s.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
    K = sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), s) for k, r in s.sinks.items())
    return s, den.to_csr(den.dense_hamiltonian(s) + shift * np.eye(s.dim)), den.to_csr(K)


@pytest.mark.parametrize("nuc,M", [([2, 3], 3), ([2] * 5, 70), ([3, 2, 2, 2, 2, 2], 33)])
@pytest.mark.parametrize("shift", [0.0, 1.0])
def test_second_pass_against_the_oracle(nuc, M, shift):
    s, H, K = _case(nuc, 41, shift)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(2.0, 0.5)
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), K_csr=K, krylov=16, nthreads=8)["traj_yield"]
    for form, prec, tol in (("streamed", "c128", 1e-10), ("resident", "c128", 1e-10), ("streamed", "c64", 1e-6)):
        assert _rel(_run(H, s, F, times, 16, prec, form, K), ref) < tol, (form, prec)


@pytest.mark.parametrize("m", [1, 4, 5, 12, 13, 20, 28, 29, 32])
def test_every_accumulator_batch(m):
    s, H, K = _case([2, 3, 2], 42, 0.0)
    F = s.trace_samples(40, 5.0)
    times = S.time_grid(40.0, 20.0)  # long steps: no Krylov vector is negligible
    ref = orc.hs_stochastic(H, F, times, h.oracle_observables(s), K_csr=K, krylov=m, nthreads=8)["traj_yield"]
    assert _rel(_run(H, s, F, times, m, "c128", "streamed", K), ref) < 1e-10
    assert _rel(_run(H, s, F, times, m, "c64", "streamed", K), ref) < 1e-5  # 20 ns steps, |H| dt about 5: FP32 rounding x 5 x m

"""Taylor and RK4 over quartet blocks (K on the electron pair) and the ensemble sums of a step.

Against the oracle's FP64 exponential and RK4 (1e-10 per trajectory), for a scalar K, unequal
sinks (K = I x K4) and a K that leaves the pair (CSR kernels), electrons not leading the basis.
"""
import numpy as np
import pytest

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from oracle import density as den
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("nuc,M", [([], 1), ([3], 65), ([2, 3, 2, 2], 33)])
@pytest.mark.parametrize("kind", ["scalar", "pair", "general"])
@pytest.mark.parametrize("propagator", ["taylor", "rk4"])
def test_against_the_oracle(nuc, M, kind, propagator):
    s = h.random_system(nuc[::2], nuc[1::2], seed=51) if nuc else \
        S.radical_pair([], [], [], [], np.array([0.0, 2e-4, 5e-5]), sink_rate=2e-3)
    K = None
    if kind != "scalar":
        s.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
        A = sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), s) for k, r in s.sinks.items())
        if kind == "general":
            A = A + 1e-3 * np.diag(np.arange(s.dim) / s.dim)
        K = den.to_csr(A)
    kappa = None if K else s.kappa()
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(3.5, 1.0) if propagator == "taylor" else S.time_grid(0.5, 0.1)
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=kappa or 0.0, K_csr=K,
                            method=1 if propagator == "taylor" else 2, nthreads=8)
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=kappa, csr=K)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(times, 1, "c128", propagator=propagator)
        per, ens = p.yields()
        values = p.values()
    assert _rel(per, ref["traj_yield"]) < 1e-10
    assert _rel(values, ref["values"]) < 1e-10 and _rel(ens, ref["yield"]) < 1e-10

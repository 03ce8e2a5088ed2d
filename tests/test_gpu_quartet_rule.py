"""Taylor and RK4 take the quartet form of H once the products asked for pay for its assembly: the
calls before, over CSR rows, and those after agree with the oracle (1e-10 per trajectory), for
several H in turn on one context.
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
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("propagator", ["taylor", "rk4"])
def test_calls_before_and_after_agree(nuc, M, pair, propagator):
    times = S.time_grid(0.2, 0.1)  # two steps: not worth the form by themselves
    with hs.HSPropagatorB200(0) as p:
        for seed in (61, 62):
            s = h.random_system(nuc[::2], nuc[1::2], seed=seed) if nuc else \
                S.radical_pair([], [], [], [], np.array([0.0, 2e-4, 5e-5 * (seed - 60)]), sink_rate=2e-3)
            K = None
            if pair:
                s.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
                K = den.to_csr(sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), s)
                                   for k, r in s.sinks.items()))
            F = s.trace_samples(M, 5.0)
            ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s),
                                    kappa=0.0 if pair else s.kappa(), K_csr=K,
                                    method=1 if propagator == "taylor" else 2, nthreads=8)
            p.set_hamiltonian(*s.hamiltonian_csr())
            p.set_reaction(kappa=None if pair else s.kappa(), csr=K)
            p.set_electron_pair(*s.electron_strides())
            p.set_observables([(op, rate) for _, op, rate in s.observables()])
            launches = []
            for _ in range(8):
                before = p.launch_count()
                p.set_factors(F)
                p.propagate(times, 1, "c128", propagator=propagator)
                launches.append(p.launch_count() - before)
                assert _rel(p.yields()[0], ref["traj_yield"]) < 1e-10
            if propagator == "taylor":  # the quartet form's sub-steps have no rescaling kernel
                assert launches[0] > launches[-1]

"""Resident complex128 form with more trajectories than one wave of its register-resident shape, at a
Krylov dimension of a few (half the warps, two rows a thread): per-trajectory yields within 1e-10 of
the oracle's Arnoldi at the edges of the shapes, with a scalar K and with unequal sinks.
"""
import numpy as np
import pytest

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from oracle import density as den
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu


# D = 36, 64, 96, 128, 144, 256, one trajectory above and at the limit of 148 (8 / warps)
@pytest.mark.parametrize("nuc,M", [([3, 3], 593), ([2] * 4, 592), ([2] * 4, 593), ([3, 2, 2, 2], 297), ([2] * 5, 297),
                                   ([3, 3, 2, 2], 149), ([2] * 6, 149)])
@pytest.mark.parametrize("m", [1, 2, 3, 6, 7])
@pytest.mark.parametrize("unequal", [False, True])
def test_many_trajectories_against_the_oracle(nuc, M, m, unequal):
    s = h.random_system(nuc[::2], nuc[1::2], seed=90 + len(nuc))
    K = None
    if unequal:
        s.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
        K = den.to_csr(sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), s) for k, r in s.sinks.items()))
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(2.0, 1.0)
    kappa = None if unequal else s.kappa()
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=kappa or 0.0, K_csr=K, krylov=m,
                            nthreads=8)
    with hs.HSPropagatorB200(0) as p:
        p.set_form("resident")
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=kappa, csr=K)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(times, m, "c128")
        per = p.yields()[0]
    assert np.max(np.abs(per - ref["traj_yield"])) / np.max(np.abs(ref["traj_yield"])) < 1e-10

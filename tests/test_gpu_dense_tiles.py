"""Dense form with whole and half trajectory tiles at ragged shapes, against the FP64-expm oracle.

A GEMM whose half tiles all fit one wave (148) takes half tiles; both accumulate in the same order, so the
shapes on either side of that limit only have to meet the forms' own error bounds per trajectory
(bf16x3 1e-4, bf16x6 1e-5, int8x4 1e-7 over 20 steps).
"""
import numpy as np
import pytest

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("bf16x3", 1e-4), ("bf16x6", 1e-5), ("int8x4", 1e-7)])
@pytest.mark.parametrize("nuc,M", [([3], 1), ([3, 2, 2], 64), ([2] * 4, 65), ([3, 3, 2], 129), ([3, 3, 3, 2], 300),
                                   ([2] * 4, 19000)])
def test_tiles_against_the_oracle(nuc, M, precision, tol):
    s = h.random_system(nuc[::2], nuc[1::2], seed=90)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(20.0, 1.0)
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=s.kappa())
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(times, 16, precision, propagator="dense")
        per = p.yields()[0]
    pick = np.unique(np.linspace(0, M - 1, 40).astype(int))  # trajectories of every tile edge region
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F[:, pick], times, h.oracle_observables(s), kappa=s.kappa(), method=1,
                            nthreads=8)["traj_yield"]
    assert np.max(np.abs(per[pick] - ref)) / np.max(np.abs(ref)) < tol

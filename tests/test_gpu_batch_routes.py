"""Batching form on every route: rows (D <= 128), quartets, the persistent launch (a basis beyond
shared memory, or D between 1536 and 2048) and back, against the oracle within 1e-6."""
import numpy as np
import pytest

from molspin_b200 import systems as S
from molspin_b200.batching import BatchB200
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu

NUCLEI = [[3], [2] * 5, [3, 3, 2, 2], [3, 3, 2, 2, 2, 2], [2] * 8, [3] + [2] * 7, [3, 3, 3, 2, 2, 2, 2]]


@pytest.mark.parametrize("ms", [(16,), (20, 7)])
def test_routes_against_the_oracle(ms):
    # m = 20 at D = 1536 leaves shared memory for the persistent launch
    times = S.time_grid(2.5, 1.0)
    systems = [h.random_system(n[::2], n[1::2], seed=70 + i, aniso=i % 2 == 0) for i, n in enumerate(NUCLEI)]
    factors = [s.trace_samples(3, 1.0 + i) for i, s in enumerate(systems)]
    for m in ms:
        with BatchB200(0) as b:
            for i, s in enumerate(systems):
                b.add(s, factors[i], seed=i)
            if m == 16:
                b.tune(times, m)
            b.run(times, m)
            for i, s in enumerate(systems):
                ref = orc.hs_stochastic(s.hamiltonian_csr(), factors[i], times, h.oracle_observables(s), kappa=s.kappa(),
                                        krylov=m, nthreads=8)
                per, _ = b.yields(i)
                err = np.max(np.abs(per - ref["traj_yield"])) / np.max(np.abs(ref["traj_yield"]))
                assert err < 1e-6, (m, NUCLEI[i], err)


def test_changing_the_krylov_dimension_changes_route_and_back():
    s = h.random_system([3] + [2] * 3, [2] * 4, seed=80)
    F = s.trace_samples(4, 2.0)
    times = S.time_grid(2.0, 1.0)
    with BatchB200(0) as b:
        b.add(s, F, seed=1)
        for m in (16, 20, 16):  # each run continues from the last one's state
            b.run(times, m)
        chained = b.yields(0)[0]
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, S.time_grid(6.0, 1.0), h.oracle_observables(s), kappa=s.kappa(),
                            krylov=16, nthreads=8)
    part = orc.hs_stochastic(s.hamiltonian_csr(), F, S.time_grid(4.0, 1.0), h.oracle_observables(s), kappa=s.kappa(),
                             krylov=16, nthreads=8)
    want = ref["traj_yield"] - part["traj_yield"]
    assert np.max(np.abs(chained - want)) / np.max(np.abs(want)) < 1e-6

"""A step's kernels are launched before their predecessors end: the order of their work must not show.

With profiling on, an event stands between every two kernels, so each starts after the one before
has ended. Both runs do the same arithmetic in the same order, so they have to agree bit for bit.
"""
import numpy as np
import pytest

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from tests import helpers as h

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nuc,M", [([2, 3], 5), ([2] * 4, 512)])
@pytest.mark.parametrize("precision,propagator", [("c128", "krylov"), ("c64", "krylov"), ("c128", "taylor"),
                                                  ("c128", "rk4"), ("bf16x3", "dense"), ("int8x4", "dense")])
@pytest.mark.parametrize("sinks", ["equal", "unequal"])
def test_early_launches_change_nothing(nuc, M, precision, propagator, sinks):
    s = h.random_system(nuc[::2], nuc[1::2], seed=77)
    K = None
    if sinks == "unequal":
        from oracle import density as den
        s.sinks = {"S": 4e-3, "T0": 1e-3, "Tp": 2e-3, "Tm": 5e-4}
        K = den.to_csr(sum(0.5 * r * den.pair_operator(S.pair_projector(S.PAIR_STATES[k]), s) for k, r in s.sinks.items()))
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(20.0, 1.0) if propagator != "rk4" else S.time_grid(2.0, 0.1)
    out = []
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=None if K else s.kappa(), csr=K)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_form("streamed")
        for profiled in (0, 1, 0):
            p.set_factors(F)
            p.profile(profiled)
            p.propagate(times, 8, precision, propagator=propagator)
            out.append((*p.yields(), p.values()))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)

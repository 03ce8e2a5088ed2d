"""GPU: a memory budget that refuses part of the quartet form leaves right results or a budget error.

The forms that can run without the quartet blocks (resident complex64, Taylor, RK4) carry on over
the rows of H.  Every budget between the set-up's memory and a whole run's is tried: two runs, a change
of coefficients and a third run equal an unlimited context's (row and quartet form: FP32 rounding of
the products, 1e-6; complex128 1e-12) or the call reports MSGPU_ERR_BUDGET.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from tests import helpers as h

pytestmark = pytest.mark.gpu
TIMES = S.time_grid(12.0, 1.0)  # enough products for Taylor and RK4 to take the quartet form


def _open(s, terms, budget=0):
    p = hs.HSPropagatorB200(0, budget)
    p.set_hamiltonian_terms(*terms, [1.0, 1e-5, 2e-5, 3e-5])
    p.set_reaction(kappa=s.kappa())
    p.set_electron_pair(*s.electron_strides())
    p.set_observables([(op, rate) for _, op, rate in s.observables()])
    return p


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("precision,propagator,tol", [("c64", "krylov", 1e-6), ("c128", "taylor", 1e-12),
                                                      ("c128", "rk4", 1e-12)])
def test_every_budget_is_right_or_refused(precision, propagator, tol):
    s = h.random_system([2, 2, 2], [2, 2, 2], seed=8)
    F, terms = s.trace_samples(4, 3.0), S.field_terms(s)

    def run(p):
        p.set_factors(F)
        p.propagate(TIMES, 12, precision, propagator=propagator)
        return p.yields()[0]

    def calls(p):  # the two runs before the coefficients change, the one after
        yield lambda: run(p)
        yield lambda: run(p)
        yield lambda: p.set_hamiltonian_coefficients([1.0, -4e-5, 1e-5, 2e-5]) or run(p)

    with _open(s, terms) as p:
        low = L.lib.msgpu_device_bytes(p.ctx)
        ref = [call() for call in calls(p)]
        high = L.lib.msgpu_device_bytes(p.ctx)
    right = refused = 0
    for budget in range(int(low), int(high) + 2048, 2048):
        try:
            p = _open(s, terms, budget)
        except hs.MsgpuError as e:
            assert e.code == L.MSGPU_ERR_BUDGET
            continue
        with p:
            for call, want in zip(calls(p), ref):
                try:
                    got = call()
                except hs.MsgpuError as e:
                    assert e.code == L.MSGPU_ERR_BUDGET
                    refused += 1
                    continue
                assert _rel(got, want) < tol, budget
                right += 1
    assert right > 3 and refused > 3

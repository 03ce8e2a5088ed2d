"""Streamed complex128 three-term recurrence at Krylov dimensions of a few and large D, where the
tiles' partial sums are bounded by the buffer that the Krylov dimension sizes: against the library's
own Arnoldi (MSGPU_REC_ARNOLDI) on the same block, within 1e-11.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from tests import helpers as h

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("nuc,M,ms", [([2] * 8 + [3, 3], 64, [1, 2]), ([2] * 12, 64, [1, 2]), ([2] * 13, 48, [1, 4])])
def test_small_krylov_dimensions_match_arnoldi(nuc, M, ms):
    s = h.random_system(nuc[:len(nuc) // 2], nuc[len(nuc) // 2:], seed=17)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(0.2, 0.1)
    csr = s.hamiltonian_csr()
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(*csr)
        p.set_reaction(kappa=s.kappa())
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        for m in ms:
            got = []
            for rec in (L.REC_AUTO, L.REC_ARNOLDI):
                p.set_factors(F)
                p.propagate(times, m, "c128", recurrence=rec)
                got.append((p.yields()[0], p.get_factors()))
            assert _rel(got[0][0], got[1][0]) < 1e-11
            assert _rel(got[0][1], got[1][1]) < 1e-11

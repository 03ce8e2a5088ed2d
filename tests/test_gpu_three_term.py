"""Streamed complex128 three-term recurrence (Hermitian H, K = kappa I) against Arnoldi and the oracle.

Per-trajectory yields within 1e-10 relative of the oracle's Arnoldi, and within 1e-11 of the
library's own Arnoldi (MSGPU_REC_ARNOLDI) on the same block.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from oracle import pyoracle as orc
from tests import helpers as h

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _run(s, F, times, m, recurrence=L.REC_AUTO, groups=0, bits=None, kappa=None):
    with hs.HSPropagatorB200(0) as p:
        p.set_form("streamed")
        p.set_option(L.OPT_TRAJ_GROUPS, groups)
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=s.kappa() if kappa is None else kappa)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        if bits is not None:
            p.set_noise(0.3, L.NOISE_REPLAY, 0, bits, len(times) - 1, F.shape[1])
        p.set_factors(F)
        p.propagate(times, m, "c128", recurrence=recurrence)
        return p.yields()[0], p.get_factors()


@pytest.mark.parametrize("nuc,M", [([], 1), ([3], 3), ([2, 3, 2], 65), ([2] * 7, 20)])
@pytest.mark.parametrize("m", [1, 2, 16, 32])
def test_small_shapes_against_the_oracle(nuc, M, m):
    s = h.random_system(nuc[::2], nuc[1::2], seed=21 + len(nuc)) if nuc else \
        S.radical_pair([], [], [], [], np.array([0.0, 2e-4, 5e-5]), sink_rate=2e-3)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(3.5, 1.0)
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=s.kappa(), krylov=m, nthreads=8)
    assert _rel(_run(s, F, times, m)[0], ref["traj_yield"]) < 1e-10


@pytest.mark.parametrize("nuc,M", [([2] * 5 + [3] * 2, 200), ([2] * 9, 520)])
def test_larger_blocks_against_arnoldi_and_across_groups(nuc, M):
    s = h.random_system(nuc[:4], nuc[4:], seed=31)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(3.0, 1.0)
    bits = np.packbits(np.random.default_rng(1).random((3, 2, M)).ravel() < 0.4, bitorder="little")
    a, xa = _run(s, F, times, 16, bits=bits)
    b, xb = _run(s, F, times, 16, recurrence=L.REC_ARNOLDI, bits=bits)
    assert _rel(a, b) < 1e-11 and _rel(xa, xb) < 1e-11
    one, x1 = _run(s, F, times, 16, groups=1, bits=bits)
    np.testing.assert_array_equal(a, one)  # groups only share out the columns
    np.testing.assert_array_equal(xa, x1)


def test_a_long_step_takes_the_pade_exponential():
    s = h.random_system([2, 2], [3], seed=11)
    F = s.trace_samples(3, 5.0)
    times = S.time_grid(4e3, 4e3)
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=1e-5, krylov=32, nthreads=8)
    # rounding of the exponential grows with dt |H| (several hundred)
    assert _rel(_run(s, F, times, 32, kappa=1e-5)[0], ref["traj_yield"]) < 4e-9

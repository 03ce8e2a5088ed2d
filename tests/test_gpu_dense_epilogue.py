"""Dense int8x4 form on both sides of the epilogue's change from 256 to 128 threads a trajectory
(592 trajectories a group of tiles): yields and values within the form's error bound (1e-7 over 10
steps) of the FP64-expm oracle, with recorded flips.
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


@pytest.mark.parametrize("nuc,M", [([3], 590), ([2] * 4, 1150), ([3, 2, 2], 1290), ([2] * 4, 1410), ([3, 3, 2, 2], 1400)])
def test_epilogue_widths_against_the_oracle(nuc, M):
    s = h.random_system(nuc[::2], nuc[1::2], seed=93)
    F = s.trace_samples(M, 5.0)
    times = S.time_grid(10.0, 1.0)
    bits = np.packbits(np.random.default_rng(3).random((10, 2, M)).ravel() < 0.3, bitorder="little")
    ref = orc.hs_stochastic(s.hamiltonian_csr(), F, times, h.oracle_observables(s), kappa=s.kappa(), method=1, nthreads=8,
                            U_csr=den.to_csr(den.st_unitary(s)), event_rate=0.15, noise_mode=1,
                            flip_bits=bits)
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=s.kappa())
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_noise(0.3, L.NOISE_REPLAY, 0, bits, 10, M)
        p.set_factors(F)
        p.propagate(times, 16, "int8x4", propagator="dense")
        per, ens = p.yields()
        values = p.values()
    assert _rel(per, ref["traj_yield"]) < 1e-7
    assert _rel(values, ref["values"]) < 1e-7 and _rel(ens, ref["yield"]) < 1e-7

"""GPU: a state that is not finite is reported, also where no observable looks.

The first trajectory has a NaN or an infinity in a T+ row of the pair; the one observable is the
singlet projector, which has no coefficient there.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from molspin_b200.batching import BatchB200
from tests import helpers as h

pytestmark = pytest.mark.gpu
TIMES = S.time_grid(2.0, 1.0)


def _block(nuclei, bad):
    s = h.random_system([2] * (nuclei // 2), [2] * (nuclei - nuclei // 2), seed=4)
    s.sinks = {"S": 1e-3}
    F = np.array(s.trace_samples(3, 2.0))
    F[0, 0] = bad  # electrons both up
    return s, F


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("nuclei", [2, 4, 6])
@pytest.mark.parametrize("form,precision", [("resident", "c128"), ("resident", "c64"), ("streamed", "c128"),
                                            ("streamed", "c64")])
def test_run_reports_it(form, precision, nuclei, bad):
    s, F = _block(nuclei, bad)
    with hs.HSPropagatorB200(0) as p:
        p.set_form(form)
        p.set_hamiltonian(*s.hamiltonian_csr())
        p.set_reaction(kappa=5e-4)
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(S.pair_projector(S.PAIR_STATES["S"]), 1e-3)])
        p.set_factors(F)
        with pytest.raises(hs.MsgpuError) as e:
            p.propagate(TIMES, 12, precision)
        assert e.value.code == L.MSGPU_ERR_NONFINITE
        p.set_factors(np.where(np.isfinite(F), F, 0.0))
        p.propagate(TIMES, 12, precision)


@pytest.mark.parametrize("nuclei", [2, 6])
def test_batch_reports_it(nuclei):
    s, F = _block(nuclei, np.nan)
    s.kappa = lambda: 5e-4
    b = BatchB200(0)
    b.add(s, F, seed=0)
    with pytest.raises(hs.MsgpuError) as e:
        b.run(TIMES, 12)
    assert e.value.code == L.MSGPU_ERR_NONFINITE

"""The allocation-free step over its routes: the resident kernel at few and at many trajectories
(short shape) and, where the basis does not fit a CTA's shared memory, the streamed kernels; each
against one step of msgpu_run (1e-12), in place as well, with non-finite input refused.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from tests import helpers as h

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nuc,M,m", [([2] * 4, 593, 3), ([3, 2, 2, 2], 297, 6), ([2] * 6, 149, 2), ([2] * 4, 593, 7),
                                     ([2], 70, 8), ([2] * 9, 20, 3)])
def test_step_against_one_run(nuc, M, m):
    import torch
    s = h.random_system(nuc[::2], nuc[1::2], seed=80 + len(nuc))
    r, c, v = s.hamiltonian_csr()
    F = s.trace_samples(M, 3.0)
    with hs.HSPropagatorB200(0) as p:
        p.set_hamiltonian(r, c, v)
        p.set_reaction(kappa=s.kappa())
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(np.array([0.0, 0.5]), m, "c128")
        ref = p.get_factors()
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (r, c, v)]
    psi = torch.from_numpy(np.ascontiguousarray(F.T)).cuda()
    out = torch.full_like(psi, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream

    def step(a, b):
        return L.lib.msgpu_krylov_step_noalloc(s.dim, dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), s.kappa(), M,
                                               a.data_ptr(), b.data_ptr(), 0.5, m, stream)

    for target in (out, psi):
        assert step(psi, target) == L.MSGPU_OK
        got = target.cpu().numpy().T
        assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-12
    psi[0, 1] = float("nan")
    assert step(psi, out) == L.MSGPU_ERR_NONFINITE

"""GPU: a batch assembles the quartet form of its systems on the device; over every form of H that
it accepts (what the device assembles and what it leaves to the host) the yields are those of a
single-system context in complex64, whose form the host assembles, to FP32 rounding (1e-6).
"""
import numpy as np
import pytest
import scipy.sparse as sp

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from molspin_b200.batching import BatchB200
from tests import helpers as h

pytestmark = pytest.mark.gpu
TIMES = S.time_grid(6.0, 1.0)


def _matrix(s):
    r, c, v = s.hamiltonian_csr()
    m = sp.csr_matrix((v, c, r), shape=(s.dim, s.dim))
    m.sum_duplicates()
    return m


def _plain(m, rng):
    return m.indptr, m.indices, m.data


def _unsorted(m, rng):
    idx = np.concatenate([a + rng.permutation(b - a) for a, b in zip(m.indptr[:-1], m.indptr[1:])])
    return m.indptr, m.indices[idx], m.data[idx]


def _repeated(m, rng):  # every entry as two halves
    ptr = 2 * m.indptr
    return ptr, np.repeat(m.indices, 2), np.repeat(0.5 * m.data, 2)


def _zeros(m, rng):  # explicit zeros far from the structure
    z = sp.csr_matrix((np.full(m.shape[0], 1e-300), (np.arange(m.shape[0]), (np.arange(m.shape[0]) * 5 + 7) % m.shape[0])),
                      shape=m.shape)
    p = (m + z).tocsr()
    p.data[np.abs(p.data) < 1e-200] = 0.0
    return p.indptr, p.indices, p.data


def _dipolar(m, rng):  # diagonal flips of one nucleus that depend on both electrons: blocks of no flip type
    n = m.shape[0]
    flip = np.arange(n) ^ 1
    e = np.where((np.arange(n) // (n // 2)) == (np.arange(n) // (n // 4)) % 2, 0.03, -0.05)
    p = (m + sp.csr_matrix((e, (np.arange(n), flip)), shape=m.shape)).tocsr()
    return p.indptr, p.indices, p.data


def _dense(m, rng):
    a = rng.normal(size=m.shape) * 0.004
    p = sp.csr_matrix(m.toarray() + a + a.T)
    return p.indptr, p.indices, p.data


FORMS = [("iso", [2] * 6, _plain), ("aniso", [2] * 6, _plain), ("aniso", [2] * 8, _plain), ("aniso", [3, 3, 2, 2], _plain),
         ("iso", [3, 2, 2, 2, 2], _plain), ("aniso", [3, 3, 3, 2, 2], _plain), ("aniso", [3] + [2] * 7, _plain),
         ("aniso", [2] * 6, _unsorted), ("aniso", [2] * 6, _repeated), ("iso", [2] * 7, _zeros), ("aniso", [2] * 6, _dipolar),
         ("aniso", [2] * 6, _dense), ("iso", [2, 2, 3, 2, 2], _unsorted)]


@pytest.mark.parametrize("m", [3, 14])
def test_batch_against_single_contexts(m):
    rng = np.random.default_rng(7)
    batch = BatchB200(0)
    want = []
    for k, (kind, nuc, form) in enumerate(FORMS):
        half = len(nuc) // 2
        s = h.random_system(nuc[:half], nuc[half:], seed=70 + k, aniso=kind == "aniso", st_rate=0.0)
        s.bilinear.append((0, 1, 0.01 * np.eye(3)))  # exchange: the own blocks are full
        csr = form(_matrix(s), rng)
        csr = (csr[0].astype(np.int32), csr[1].astype(np.int32), np.asarray(csr[2], np.complex128))
        F = s.trace_samples(3 + k, 2.0 + k)
        kappa, strides = s.kappa(), s.electron_strides()
        with hs.HSPropagatorB200(0) as p:
            p.set_hamiltonian(*csr)
            p.set_reaction(kappa=kappa)
            p.set_electron_pair(*strides)
            p.set_observables([(op, rate) for _, op, rate in s.observables()])
            p.set_factors(F)
            p.propagate(TIMES, m, "c64")
            want.append(p.yields()[0])
        s.hamiltonian_csr = lambda v=csr: v
        batch.add(s, F, seed=k)
    batch.run(TIMES, m)
    for k, ref in enumerate(want):
        got = batch.yields(k)[0]
        assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-6, FORMS[k]

"""GPU: Hamiltonian terms whose blocks coincide in one combination and not in another.

Nucleus a has coupling J in terms 0 and 2, nucleus b has 2J in term 1: a combination with weights
w0 + w2 = 2 w1 gives both the same flip blocks, the coefficients (1, 1, 0) do not.  Every form is
compared with a context that holds the combined H: 1e-12 relative per trajectory in complex128 (the
combination differs in summation order only), 1e-7 in complex64 (the same H rounded the same way).
The same for one nucleus whose flip blocks depend on the second electron in such terms: they are the
same for both of its states in that combination alone.
"""
import numpy as np
import pytest
import scipy.sparse as sp

from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S

pytestmark = pytest.mark.gpu
J = 0.5  # a power of two: the combination of the two terms rounds as the one term does


def _system(couplings, field=False):
    """Two electrons and six spin-1/2 nuclei; couplings: {nucleus: J} to the first electron."""
    s = S.SpinSystem(mult=[2] * 8, names=["E1", "E2"] + [f"N{k}" for k in range(6)], electrons=(0, 1))
    for k, j in couplings.items():
        s.bilinear.append((0, 2 + k, j * np.eye(3)))
    if field:
        s.linear += [(0, np.array([0.02, 0.05, 0.8])), (1, np.array([-0.03, 0.04, 0.7]))]
    s.sinks = {k: 1e-3 for k in ("S", "T0", "Tp", "Tm")}
    return s


def _terms():
    rest = _system({2: 0.21, 3: -0.4, 4: 0.33, 5: 0.11}, field=True)
    return (rest, *_pattern([_matrix(s) for s in (_system({0: J}), _system({1: 2 * J}), _system({0: J}), rest)]))


def _terms_second_electron():
    rest = _system({2: 0.21, 3: -0.4, 4: 0.33, 5: 0.11}, field=True)
    sx = sp.csr_matrix(np.array([[0.0, 0.5], [0.5, 0.0]]))

    def flip(j, up):  # j S_x(E1) I_x(N0), for one state of the second electron
        e2 = sp.csr_matrix(np.diag([1.0, 0.0] if up else [0.0, 1.0]))
        return sp.kron(sp.kron(sp.kron(j * sx, e2), sx), sp.identity(32)).tocsr()

    return (rest, *_pattern([flip(J, True), flip(2 * J, False), flip(J, True), _matrix(rest)]))


def _matrix(s):
    r, c, v = s.hamiltonian_csr()
    m = sp.csr_matrix((v, c, r), shape=(256, 256))
    m.sum_duplicates()
    return m


def _pattern(mats):
    pat = sum(abs(m) for m in mats).tocsr()
    pat.sort_indices()
    rows = np.repeat(np.arange(256), np.diff(pat.indptr))
    vals = np.stack([np.asarray(m[rows, pat.indices]).ravel() for m in mats]).astype(np.complex128)
    return pat.indptr.astype(np.int32), pat.indices.astype(np.int32), vals


def _run(p, s, F, precision, propagator):
    p.set_reaction(kappa=s.kappa())
    p.set_electron_pair(*s.electron_strides())
    p.set_observables([(op, rate) for _, op, rate in s.observables()])
    p.set_factors(F)
    p.propagate(S.time_grid(12.0, 1.0), 14, precision, propagator=propagator)
    return p.yields()[0]


@pytest.mark.parametrize("terms", [_terms, _terms_second_electron])
@pytest.mark.parametrize("form,precision,propagator,tol", [
    ("resident", "c64", "krylov", 1e-7), ("streamed", "c64", "krylov", 1e-7), ("streamed", "c128", "krylov", 1e-12),
    ("auto", "c128", "taylor", 1e-12), ("auto", "c128", "rk4", 1e-12)])
def test_coinciding_blocks_follow_their_own_terms(form, precision, propagator, tol, terms):
    s, r, c, vals = terms()
    F = s.trace_samples(33, 2.0)
    with hs.HSPropagatorB200(0) as p:
        p.set_form(form)
        p.set_hamiltonian_terms(r, c, vals, [1.0, 0.5, 1.0, 1.0])
        _run(p, s, F, precision, propagator)
        for coef in ([1.0, 1.0, 0.0, 1.0], [0.3, 1.0, 0.2, 0.9]):
            p.set_hamiltonian_coefficients(coef)
            got = _run(p, s, F, precision, propagator)
            with hs.HSPropagatorB200(0) as q:
                q.set_form(form)
                q.set_hamiltonian(r, c, np.tensordot(coef, vals, 1))
                ref = _run(q, s, F, precision, propagator)
            assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < tol

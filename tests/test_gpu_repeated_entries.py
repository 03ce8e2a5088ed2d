"""GPU: a Hamiltonian whose CSR rows hold a column more than once stands for the sum.

Every entry is given as three parts, apart in its row.  Against the merged matrix: 1e-12 relative in
complex128 (the parts' sum rounds once more), 1e-6 in complex64 (the merged values may round to the
next FP32 number).  One that is Hermitian entry by entry but not in its sums runs Arnoldi.
"""
import numpy as np
import pytest

from molspin_b200 import _lib as L
from molspin_b200 import hsgeneral as hs
from molspin_b200 import systems as S
from tests import helpers as h

pytestmark = pytest.mark.gpu


def _split(r, c, v):
    """Each entry as parts 1/4, 1/2 and 1/4 of it (exact), all firsts of a row before its seconds."""
    ptr, col, val = [0], [], []
    for k in range(len(r) - 1):
        a, b = r[k], r[k + 1]
        for part in (0.25, 0.5, 0.25):
            col.extend(c[a:b])
            val.extend(part * v[..., a:b].T)
        ptr.append(len(col))
    return np.array(ptr, np.int32), np.array(col, np.int32), np.ascontiguousarray(np.array(val).T)


def _run(s, F, upload, precision, propagator="krylov", form="auto", recurrence=L.REC_AUTO, m=12):
    with hs.HSPropagatorB200(0) as p:
        p.set_form(form)
        upload(p)
        p.set_reaction(kappa=s.kappa())
        p.set_electron_pair(*s.electron_strides())
        p.set_observables([(op, rate) for _, op, rate in s.observables()])
        p.set_factors(F)
        p.propagate(S.time_grid(12.0, 1.0) if m > 4 else S.time_grid(16.0, 8.0), m, precision, propagator=propagator, recurrence=recurrence)
        return p.yields()[0]


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("form,precision,propagator,tol", [
    ("resident", "c64", "krylov", 1e-6), ("streamed", "c64", "krylov", 1e-6), ("streamed", "c128", "krylov", 1e-12),
    ("auto", "c128", "taylor", 1e-12), ("auto", "c128", "rk4", 1e-12)])
def test_parts_add_up(form, precision, propagator, tol):
    s = h.random_system([2, 2, 2], [2, 2, 2], seed=5)
    F = s.trace_samples(9, 3.0)
    r, c, v = S.field_terms(s)
    coef = [1.0, 2e-5, -3e-5, 4e-5]
    merged = np.tensordot(coef, v, 1)
    ref = _run(s, F, lambda p: p.set_hamiltonian(r, c, merged), precision, propagator, form)
    got = _run(s, F, lambda p: p.set_hamiltonian(*_split(r, c, merged)), precision, propagator, form)
    assert _rel(got, ref) < tol
    got = _run(s, F, lambda p: p.set_hamiltonian_terms(*_split(r, c, v), coef), precision, propagator, form)
    assert _rel(got, ref) < tol


@pytest.mark.parametrize("form", ["resident", "streamed"])
def test_sums_that_are_not_hermitian_run_arnoldi(form):
    s = h.random_system([2, 2], [2, 2], seed=6)
    F = s.trace_samples(5, 3.0)
    r, c, v = s.hamiltonian_csr()
    # the largest off-diagonal entry of a row twice, its transpose once: each has a partner, the sums differ
    row = 20
    k = max(range(r[row], r[row + 1]), key=lambda i: abs(v[i]) * (c[i] != row))
    ptr = np.concatenate([r[:row + 1], r[row + 1:] + 1]).astype(np.int32)
    col, val = np.insert(c, r[row + 1], c[k]).astype(np.int32), np.insert(v, r[row + 1], v[k])
    up = lambda p: p.set_hamiltonian(ptr, col, val)  # noqa: E731
    a = _run(s, F, up, "c128", form=form, m=4)
    b = _run(s, F, up, "c128", form=form, recurrence=L.REC_ARNOLDI, m=4)
    # (four vectors do not hold a step of 8 ns, so the recurrences differ where H is not Hermitian)
    assert _rel(a, b) < 1e-12

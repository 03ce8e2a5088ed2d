"""Benchmark cases of the propagation library, from the smallest call to the largest.

Every case is work that a program hands to the library through its public entry points: the
allocation-free step of the C ABI, ``HSPropagatorB200`` (Krylov, dense, Taylor and RK4 propagators,
field terms) and ``BatchB200``.  The shapes are those of ``molspin_b200.systems``: radical pairs of
two electrons and spin-1/2 or spin-1 nuclei, trace-sampled singlet starts, dt of 0.5 or 1 ns.

A pass of a case uploads the trajectory block (from device memory, as a program that draws its
samples there does), propagates it over the whole time grid and reads the yields back.  The
forms that hold their vectors in 32 bits or fewer (complex64, the BF16 splits) return their results
as 32-bit values, the others in 64 bits.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from molspin_b200 import _lib as L
from molspin_b200 import systems as S
from molspin_b200.batching import BatchB200
from molspin_b200.hsgeneral import HSPropagatorB200

MU = 8.79410005e1  # rad / (ns T)
G_E = 2.0023


def listed():
    return [
        # One step for a host that owns all device memory (the 16 MiB scratch area): the smallest call.
        dict(name="noalloc-d64", kind="noalloc", nuc="2222", m=16, M=64, dt=1.0),
        # The plain configuration: 4 spin-1/2 nuclei, 256 samples, complex128.
        dict(name="plain-d64", kind="system", nuc="2222", m=16, M=256, steps=100, dt=1.0, prec="c128", prop="krylov",
             noise="none", sinks="equal", state=True),
        # Uneven little system of a relaxation study: a spin-1 nucleus, unequal sinks, the reference's flip bits.
        dict(name="sinks-d96", kind="system", nuc="3222", m=16, M=100, steps=50, dt=1.0, prec="c128", prop="krylov",
             noise="replay", sinks="unequal", state=True),
        # Field sweep (powder or MARY curve) of a mid-size pair on one context: two directions, complex64.
        dict(name="sweep-d1024", kind="sweep", nuc="22222222", m=16, M=256, steps=20, dt=1.0, prec="c64",
             prop="krylov", noise="philox", sinks="equal", fields=2, state=False),
        # A request of the serving mix above the persistent route, spin-1 nuclei, ragged trajectory count.
        dict(name="request-d9216", kind="system", nuc="2222222233", m=16, M=250, steps=20, dt=1.0, prec="c64",
             prop="krylov", noise="philox", sinks="equal", state=False),
        # The precision configuration: 12 nuclei, 1024 trajectories, m = 20, complex64.  The headline workload.
        dict(name="precision-d16384", kind="system", nuc="222222222222", m=20, M=1024, steps=20, dt=0.5, prec="c64",
             prop="krylov", noise="none", sinks="equal", state=False),
        # The same Hamiltonian size in the reference-parity precision.
        dict(name="plain-d16384", kind="system", nuc="222222222222", m=20, M=512, steps=4, dt=0.5, prec="c128",
             prop="krylov", noise="none", sinks="equal", state=False),
        # Unequal sinks in complex64 (Arnoldi on the electron-pair reaction operator).
        dict(name="sinks-d4096", kind="system", nuc="2222222222", m=16, M=256, steps=10, dt=1.0, prec="c64",
             prop="krylov", noise="none", sinks="unequal", state=False),
        # Dense tensor-core propagator: the 4096-trajectory configuration.
        dict(name="dense-d1024", kind="system", nuc="22222222", m=16, M=4096, steps=50, dt=1.0, prec="bf16x3",
             prop="dense", noise="none", sinks="equal", state=False),
        # Dense propagator with exact accumulation on a ragged shape.
        dict(name="dense-d576", kind="system", nuc="222233", m=16, M=1000, steps=50, dt=1.0, prec="int8x4",
             prop="dense", noise="replay", sinks="equal", state=False),
        # The reference's autoexpm propagator.
        dict(name="taylor-d2048", kind="system", nuc="222222222", m=1, M=256, steps=5, dt=1.0, prec="c128",
             prop="taylor", noise="none", sinks="equal", state=False),
        # Batching form: many uneven pairs propagated together (a parameter scan).
        dict(name="batch-16", kind="batch", systems=16, scan=1, nmin=4, nmax=10, m=16, mmax=512, steps=20, dt=1.0),
    ]


def draw(rng: random.Random):
    """One more case of the same ranges, no dearer than the largest listed one."""
    def cost(c):
        """Vector traffic of the Krylov, Taylor and RK4 forms; the dense form is bounded by its sizes."""
        if c["kind"] in ("noalloc", "batch") or c["prop"] == "dense":
            return 0
        small = _dim(c["nuc"]) <= 1024
        return (_dim(c["nuc"]) * c["M"] * c["steps"] * c["m"] * c.get("fields", 1) * (40 if small else 1) *
                (2 if c["prec"] == "c64" and c["sinks"] == "equal" else 10))

    big = [c for c in listed() if c["name"] == "precision-d16384"]
    cap = cost(big[0])

    def nuclei(lo, hi, dmax):
        while True:
            n = rng.randint(lo, hi)
            ones = rng.choice([0, 0, 1, 2])
            s = "2" * max(0, n - ones) + "3" * min(n, ones)
            if _dim(s) <= dmax:
                return s

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["noalloc", "resident", "resident", "sweep", "streamed", "streamed", "plain", "sinks", "dense",
                       "dense", "series", "series", "batch"])
    while True:
        if kind == "noalloc":
            c = dict(kind="noalloc", nuc=nuclei(2, 4, 150), m=rng.randint(8, 16), M=size(4, 128), dt=1.0)
        elif kind == "batch":
            c = dict(kind="batch", systems=rng.randint(4, 16), scan=rng.randint(2, 9999), nmin=4,
                     nmax=rng.randint(6, 10), m=16, mmax=size(64, 512), steps=rng.randint(10, 20), dt=1.0)
        else:
            c = dict(kind="system", dt=rng.choice([0.5, 1.0]), noise=rng.choice(["none", "replay", "philox"]),
                     sinks="equal", prop="krylov", m=rng.randint(12, 20), state=False)
            if kind in ("resident", "sweep"):
                c.update(nuc=nuclei(2, 8, 1024), M=size(5, 1024), steps=rng.randint(20, 100),
                         prec=rng.choice(["c128", "c64"]), sinks="equal")
                if kind == "sweep":
                    c.update(kind="sweep", fields=rng.randint(2, 4))
                elif c["prec"] == "c128":
                    c.update(sinks=rng.choice(["equal", "unequal"]), state=True)
            elif kind == "streamed":
                c.update(nuc=nuclei(9, 14, 65536), M=size(48, 1024), steps=rng.randint(4, 20), prec="c64")
            elif kind == "plain":
                c.update(nuc=nuclei(9, 12, 16384), M=size(48, 512), steps=rng.randint(2, 4), prec="c128")
            elif kind == "sinks":
                c.update(nuc=nuclei(9, 11, 9216), M=size(48, 512), steps=rng.randint(4, 10), prec="c64",
                         sinks="unequal")
            elif kind == "dense":
                c.update(nuc=nuclei(4, 8, 1024), M=size(200, 4096), steps=rng.randint(20, 50),
                         prec=rng.choice(["bf16x3", "bf16x6", "int8x4"]), prop="dense",
                         sinks=rng.choice(["equal", "equal", "unequal"]))
            else:
                c.update(nuc=nuclei(5, 9, 2304), M=size(48, 512), steps=rng.randint(2, 5), prec="c128", m=1,
                         prop=rng.choice(["taylor", "rk4"]), dt=0.5, sinks=rng.choice(["equal", "unequal"]))
        if cost(c) <= cap:
            return c


def _dim(nuc: str) -> int:
    return 4 * math.prod(int(ch) for ch in nuc)


def _batch_shapes(case):
    """(nuclei, trajectories) of a batch's systems; a fixed list per case, as a scan's input file is."""
    rng = random.Random(case["scan"])
    out = []
    for k in range(case["systems"]):
        # every nucleus count of the range in turn, so that each route of the batch has work
        n = case["nmin"] + k % (case["nmax"] - case["nmin"] + 1)
        ones = rng.randint(0, 2)
        out.append(("2" * (n - ones) + "3" * ones, rng.randint(min(64, case["mmax"]), case["mmax"])))
    return out


# ------------------------------------------------------------------ inputs
def _numbers(nuc: str, seed: int, iso: bool = False):
    """Couplings (mT), field (T), sink rates and dephasing rate of one radical pair."""
    rng = np.random.default_rng(seed)
    half = (len(nuc) + 1) // 2
    A = []
    for _ in nuc:
        if iso:
            A.append(np.eye(3) * rng.uniform(-1.0, 1.0))
        else:
            q, _r = np.linalg.qr(rng.normal(size=(3, 3)))
            A.append(q @ np.diag(rng.uniform(-1.5, 1.5, size=3)) @ q.T)
    A = [0.5 * (a + a.T) for a in A]
    d = rng.normal(size=3)
    d /= np.linalg.norm(d)
    return dict(half=half, A=A, B=50e-6 * d, rates=rng.uniform(0.5e-3, 2e-3, size=4), st=5e-3, iso=iso)


def _system(nuc: str, num, sinks: str):
    mult = [int(ch) for ch in nuc]
    h = num["half"]
    s = S.radical_pair(mult[:h], mult[h:], num["A"][:h], num["A"][h:], num["B"], sink_rate=float(num["rates"][0]))
    if sinks == "unequal":
        s.sinks = {k: float(r) for k, r in zip(("S", "T0", "Tp", "Tm"), num["rates"])}
    return s


def _pair_reaction(s) -> np.ndarray:
    """K on the electron pair: sum_c k_c / 2 P_c."""
    return sum(0.5 * r * S.pair_projector(S.PAIR_STATES[k]) for k, r in s.sinks.items())


def _reaction_csr(s):
    k4, Z = _pair_reaction(s), s.dim // 4
    rows, cols, vals = [], [], []
    for a in range(4):
        b = np.flatnonzero(np.abs(k4[a]) > 0)
        rows.append(np.full(Z, len(b)))
        cols.append((b[None, :] * Z + np.arange(Z)[:, None]).ravel())
        vals.append(np.tile(k4[a][b], Z))
    ptr = np.concatenate([[0], np.cumsum(np.concatenate(rows))])
    return ptr.astype(np.int32), np.concatenate(cols).astype(np.int32), np.concatenate(vals)


def _factors(D: int, M: int, seed: int) -> torch.Tensor:
    """Singlet pair times random nuclear states over sqrt(M), M x D on the GPU (a trajectory per row)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    chi = torch.randn(M, D // 4, 2, dtype=torch.float64, device="cuda", generator=g)
    chi = torch.view_as_complex(chi / chi.square().sum(dim=(1, 2), keepdim=True).sqrt())
    pair = torch.tensor([0.0, 1.0, -1.0, 0.0], dtype=torch.complex128, device="cuda") / math.sqrt(2.0)
    return (pair[None, :, None] * chi[:, None, :]).reshape(M, D).contiguous() / math.sqrt(M)


def _flip_bits(case, num, seed: int) -> np.ndarray:
    """Flip decisions (steps, 2, M) of the singlet-triplet dephasing, as a recorded stream."""
    p = -0.5 * math.expm1(-num["st"] * 0.5 * case["dt"])
    return np.random.default_rng(seed + 7).random((case["steps"], 2, case["M"])) < p


def _check(ctx, rc):
    if rc:
        raise RuntimeError(L.lib.msgpu_last_error(ctx).decode())


class _Held:
    """What a program keeps between calls: the context and its inputs."""


def prepare(case, seed: int):
    st = _Held()
    st.case = case
    if case["kind"] == "batch":
        st.times = np.arange(case["steps"] + 1) * case["dt"]
        st.batch = BatchB200(0)
        for k, (nuc, M) in enumerate(_batch_shapes(case)):
            s = _system(nuc, _numbers(nuc, 1000 * seed + k, iso=True), "equal")
            st.batch.add(s, _factors(s.dim, M, 1000 * seed + k).T.cpu().numpy(), seed=k)
        return st
    num = _numbers(case["nuc"], seed)
    s = _system(case["nuc"], num, case.get("sinks", "equal"))
    st.F = _factors(s.dim, case["M"], seed)
    if case["kind"] == "noalloc":
        r, c, v = s.hamiltonian_csr()
        st.csr = [torch.from_numpy(x).cuda() for x in (r, c, v)]
        st.kappa, st.out = s.kappa(), torch.empty_like(st.F)
        return st
    st.times = np.arange(case["steps"] + 1) * case["dt"]
    p = st.p = HSPropagatorB200(0)
    if case["kind"] == "sweep":
        p.set_hamiltonian_terms(*S.field_terms(s), [1.0, *num["B"]])
        st.fields = _fields(case, num)
    else:
        p.set_hamiltonian(*s.hamiltonian_csr())
    if case["sinks"] == "equal":
        p.set_reaction(kappa=s.kappa())
    else:
        p.set_reaction(csr=_reaction_csr(s))
    p.set_electron_pair(*s.electron_strides())
    p.set_observables([(op, rate) for _, op, rate in s.observables()])
    if case["noise"] == "replay":
        bits = np.packbits(_flip_bits(case, num, seed).ravel(), bitorder="little")
        p.set_noise(num["st"], L.NOISE_REPLAY, 0, bits, case["steps"], case["M"])
    elif case["noise"] == "philox":
        p.set_noise(num["st"], L.NOISE_PHILOX, seed)
    return st


def _fields(case, num):
    """Fields of a sweep: the system's own direction, then others of growing strength."""
    return [num["B"] * (1.0 + k) * (-1.0) ** k for k in range(case["fields"])]


# ------------------------------------------------------------------ one pass
def _upload(st):
    p, F = st.p, st.F
    _check(p.ctx, L.lib.msgpu_upload_factors_device(p.ctx, F.shape[1], F.shape[0], ctypes.c_void_p(F.data_ptr())))
    p.M = F.shape[0]


def _results(st):
    p, case = st.p, st.case
    per, ens = p.yields()
    out = {"traj_yields": per, "yields": ens, "values": p.values()}
    if case["state"]:
        out["state"] = p.get_factors()
    if case["prec"] in ("c64", "bf16x3", "bf16x6"):
        out = {k: v.astype(np.complex64 if v.dtype.kind == "c" else np.float32) for k, v in out.items()}
    return out


def run(st):
    case = st.case
    if case["kind"] == "noalloc":
        r, c, v = st.csr
        pi, pd = ctypes.POINTER(ctypes.c_int), ctypes.c_void_p
        rc = L.lib.msgpu_krylov_step_noalloc(st.F.shape[1], pd(r.data_ptr()), pd(c.data_ptr()), pd(v.data_ptr()),
                                             st.kappa, st.F.shape[0], pd(st.F.data_ptr()), pd(st.out.data_ptr()),
                                             case["dt"], case["m"],
                                             pd(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(f"msgpu_krylov_step_noalloc: {rc}")
        return st.out
    if case["kind"] == "batch":
        st.batch.run(st.times, case["m"])
        got = [st.batch.yields(k) for k in range(case["systems"])]
        return {"traj_yields": [a.astype(np.float32) for a, _ in got], "yields": [b.astype(np.float32) for _, b in got]}
    if case["kind"] == "sweep":
        out = []
        for B in st.fields:
            st.p.set_hamiltonian_coefficients([1.0, *B])
            _upload(st)
            st.p.propagate(st.times, case["m"], case["prec"])
            out.append(_results(st))
        return out
    _upload(st)
    st.p.propagate(st.times, case["m"], case["prec"], propagator=case["prop"])
    return _results(st)


# ------------------------------------------------------------------ work
def _nnz(nuc: str, iso: bool) -> int:
    """Nonzeros of H: the diagonal, the two electron flips, and per nucleus its flips with (isotropic
    couplings: only opposite to) the electron's."""
    return int(_dim(nuc) * (3 + sum(2.0 * (int(ch) - 1) / int(ch) * (0.5 if iso else 2.0) for ch in nuc)))


def _step_work(D, M, m, nnz, prop, prec):
    if prop == "dense":
        products = {"bf16x3": 3, "bf16x6": 6, "int8x4": 10}[prec]
        return 8.0 * D * D * M * products
    if prop == "taylor":
        return 20 * 8.0 * nnz * M
    if prop == "rk4":
        return 4 * 8.0 * nnz * M
    # Krylov: m products with H, m dot products and vector updates, the final combination
    return M * (m * 8.0 * nnz + m * 24.0 * D + m * 8.0 * D)


def work(case):
    if case["kind"] == "batch":
        flops = sum(case["steps"] * _step_work(_dim(n), M, case["m"], _nnz(n, True), "krylov", "c64")
                    for n, M in _batch_shapes(case))
        return {"bytes": sum(16.0 * _dim(n) * M + 12.0 * _nnz(n, True) for n, M in _batch_shapes(case)),
                "flops": flops}
    D, M, nnz = _dim(case["nuc"]), case["M"], _nnz(case["nuc"], False)
    if case["kind"] == "noalloc":
        return {"bytes": 2 * 16.0 * D * M + 20.0 * nnz, "flops": _step_work(D, M, case["m"], nnz, "krylov", "c128")}
    f = _step_work(D, M, case["m"], nnz, case["prop"], case["prec"])
    n = case.get("fields", 1)
    return {"bytes": n * (16.0 * D * M + 20.0 * nnz + 8.0 * 4 * (M + case["steps"])), "flops": n * case["steps"] * f}


# ------------------------------------------------------------------ 64-bit values
def _spin(d: int):
    s = (d - 1) / 2.0
    m = s - np.arange(d)
    plus = np.zeros((d, d))
    for k in range(d - 1):
        plus[k, k + 1] = math.sqrt(s * (s + 1) - m[k + 1] * (m[k + 1] + 1))
    return [0.5 * (plus + plus.T) + 0j, -0.5j * (plus - plus.T), np.diag(m) + 0j]


def _hamiltonian(nuc: str, num, field) -> torch.Tensor:
    """H as a sparse matrix, from Kronecker products of spin matrices."""
    mult = [2, 2] + [int(ch) for ch in nuc]
    D = math.prod(mult)
    strides = [math.prod(mult[k + 1:]) for k in range(len(mult))]
    idx = np.arange(D)
    rows, cols, vals = [], [], []

    def add(sites, mat):
        """mat acts on the given sites, identity elsewhere."""
        dims = [mult[k] for k in sites]
        here = np.zeros(D, dtype=np.int64)
        for k in sites:
            here = here * mult[k] + idx // strides[k] % mult[k]
        for a, b in zip(*np.nonzero(np.abs(mat) > 0)):
            r = idx[here == a]
            shift, aa, bb = 0, int(a), int(b)
            for k, d in zip(reversed(sites), reversed(dims)):
                shift += (bb % d - aa % d) * strides[k]
                aa, bb = aa // d, bb // d
            rows.append(r)
            cols.append(r + shift)
            vals.append(np.full(len(r), mat[a, b]))

    for e in (0, 1):
        add([e], sum(MU * G_E * field[a] * _spin(2)[a] for a in range(3)))
    for n, A in enumerate(num["A"]):
        e, d = (0 if n < num["half"] else 1), mult[2 + n]
        add([e, 2 + n], sum(MU * 1e-3 * G_E * A[a, b] * np.kron(_spin(2)[a], _spin(d)[b])
                            for a in range(3) for b in range(3)))
    t = torch.sparse_coo_tensor(np.stack([np.concatenate(rows), np.concatenate(cols)]), np.concatenate(vals), (D, D))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return t.to(dev).coalesce()  # duplicates add up


def _philox_flips(seed: int, steps: int, M: int, p: float) -> np.ndarray:
    """Philox4x32-10 (Salmon et al., SC'11) keyed by the seed, counter (trajectory, step, half, tag)."""
    t, s, h = np.meshgrid(np.arange(M), np.arange(steps), np.arange(2), indexing="ij")
    c = [x.astype(np.uint64) for x in (t, s, h, np.full_like(t, 0x53544E31))]
    k0, k1, mask = seed & 0xFFFFFFFF, seed >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & mask, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = ((c[0] >> np.uint64(5)) << np.uint64(26)) | (c[1] >> np.uint64(6))
    return (u.astype(np.float64) / 2.0 ** 53 < p).transpose(1, 2, 0)


def _exact_yields(nuc, num, sinks, field, F, steps, dt, flips):
    """Yields, values and final state by the matrix exponential of every step (dense up to D = 1024,
    a converged Taylor series on the sparse matrix above)."""
    H = _hamiltonian(nuc, num, field)
    D, M = _dim(nuc), F.shape[0]
    Z = D // 4
    r = num["rates"] if sinks == "unequal" else np.full(4, num["rates"][0])
    proj = [S.pair_projector(S.PAIR_STATES[k]) for k in ("S", "T0", "Tp", "Tm")]
    dev, cd = F.device, torch.complex128
    ops = torch.tensor(np.stack([rate * P for rate, P in zip(r, proj)]), dtype=cd, device=dev)
    K4 = torch.tensor(sum(0.5 * rate * P for rate, P in zip(r, proj)), dtype=cd, device=dev)
    U4 = torch.tensor(2 * proj[0] - np.eye(4), dtype=cd, device=dev)
    x = F.T.contiguous()
    if D <= 1024:
        G = -1j * H.to_dense() - torch.kron(K4, torch.eye(Z, dtype=cd, device=dev))
        E = torch.linalg.matrix_exp(dt * G)
        step = lambda v: E @ v  # noqa: E731
    else:
        Hs = H.to_sparse_csr()
        norm = dt * (float(torch.sparse.sum(H.abs(), dim=1).to_dense().max()) + float(r.max()))
        sub = max(1, math.ceil(norm / 2.0))

        def apply(v):
            return -1j * (Hs @ v) - (K4 @ v.reshape(4, Z * M)).reshape(D, M)

        def step(v):
            for _ in range(sub):
                term, acc = v, v.clone()
                for k in range(1, 25):
                    term = apply(term) * (dt / sub / k)
                    acc += term
                v = acc
            return v

    def flip(v, mask):
        if not mask.any():
            return v
        w = v.reshape(4, Z, M)
        m = torch.from_numpy(np.ascontiguousarray(mask)).to(dev)
        return torch.where(m[None, None, :], (U4 @ w.reshape(4, Z * M)).reshape(4, Z, M), w).reshape(D, M)

    def observe(v):
        w = v.reshape(4, Z, M)
        rho = torch.einsum("azm,bzm->mab", w, w.conj())
        return torch.einsum("oab,mba->mo", ops, rho).real

    val = [observe(x)]
    for s in range(steps):
        if flips is not None:
            x = flip(x, flips[s, 0])
        x = step(x)
        if flips is not None:
            x = flip(x, flips[s, 1])
        val.append(observe(x))
    v = torch.stack(val)
    per = dt * (v[:-1] + v[1:]).sum(0) / 2
    return per, per.sum(0), v.sum(1), x


def exact(case, seed: int):
    if case["kind"] == "batch":
        per, ens = [], []
        for k, (nuc, M) in enumerate(_batch_shapes(case)):
            F = _factors(_dim(nuc), M, 1000 * seed + k)
            a, b, _v, _x = _exact_yields(nuc, n := _numbers(nuc, 1000 * seed + k, iso=True), "equal", n["B"], F,
                                         case["steps"], case["dt"], None)
            per.append(a)
            ens.append(b)
        return {"traj_yields": per, "yields": ens}
    num = _numbers(case["nuc"], seed)
    F = _factors(_dim(case["nuc"]), case["M"], seed)
    if case["kind"] == "noalloc":
        return _exact_yields(case["nuc"], num, "equal", num["B"], F, 1, case["dt"], None)[3].T.contiguous()
    if case["prop"] == "rk4":
        return None  # an explicit method: its own error is far above rounding
    flips = None
    if case["noise"] == "replay":
        flips = _flip_bits(case, num, seed)
    elif case["noise"] == "philox":
        flips = _philox_flips(seed, case["steps"], case["M"], -0.5 * math.expm1(-num["st"] * 0.5 * case["dt"]))
    out = []
    for B in _fields(case, num) if case["kind"] == "sweep" else [num["B"]]:
        per, ens, val, x = _exact_yields(case["nuc"], num, case["sinks"], B, F, case["steps"], case["dt"], flips)
        o = {"traj_yields": per, "yields": ens, "values": val}
        if case["state"]:
            o["state"] = x
        out.append(o)
    return out if case["kind"] == "sweep" else out[0]

"""Performance cases: the operator applications a program makes on the GPU.

Every case goes through the Python front end over the C ABI (``mul_``,
``mul_super``, ``Batch``, ``rk4``) with device-resident states, as an ODE
right-hand side, a master-equation solver or a sweep over models calls it.  A
case names a family, its sizes and an arithmetic form:

* ``"c128"``  ComplexF64, ``"c64"`` ComplexF32, ``"ff"`` ComplexF64 data
  applied in double-float arithmetic (``arith="ff"``).

Operators carry parameters drawn from the seed; states are seeded random kets
(normalised columns).  ``exact`` restates each family in 64 bits with torch
alone: site matrices applied one by one, dense products, ``torch.fft``.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "quantumopticsbase.jl_gb300"))

import qobgpu as Q  # noqa: E402
from qobgpu import _lib as L  # noqa: E402
from qobgpu import evolution as EV  # noqa: E402
from qobgpu import superoperators as SO  # noqa: E402
from qobgpu.bases import MomentumBasis, PositionBasis  # noqa: E402
from qobgpu.device import prepare as compile_op  # noqa: E402
from qobgpu.mul import mul_  # noqa: E402
from qobgpu.particle import potentialoperator, transform  # noqa: E402

FORMS = ("c128", "c64", "ff")


def listed():
    return [
        # One small system, one state: the right-hand side of a Schroedinger
        # equation of the two-cavity Jaynes-Cummings model (512 states), where
        # the latency of a call counts.
        dict(name="jc_ket", family="jc", n1=15, n2=15, kets=1, form="c128"),
        # The headline workload: 14-spin Heisenberg chain on a batch of 64 kets.
        dict(name="chain14_kets64", family="chain", spins=14, kets=64, form="c128"),
        # A larger chain in single precision on an odd number of kets.
        dict(name="chain16_kets51_f32", family="chain", spins=16, kets=51, form="c64"),
        # One large state (2^20 amplitudes) in double-float arithmetic.
        dict(name="chain20_ket_ff", family="chain", spins=20, kets=1, form="ff"),
        # Master equation: the lazy Liouvillian of a decaying 10-spin chain on a
        # 1024 x 1024 density operator.
        dict(name="lindblad10", family="lindblad", spins=10, form="c128"),
        # sparse(H) of the 32 x 2 x 64 Jaynes-Cummings model on 251 columns of a
        # density operator (an odd number).
        dict(name="sparse_columns", family="sparse", n1=31, n2=63, kets=251, form="c128"),
        # rho * H: an operator from the right, on the rows of a 1000 x 1024 operator.
        dict(name="rows_times_chain10", family="rows", spins=10, rows=1000, form="c128"),
        # A dense operator (no structure known) on 16 kets, single precision.
        dict(name="dense4096_kets16_f32", family="dense", n=4096, kets=16, form="c64"),
        # Mode products of dense LazyTensor factors (ragged sizes) on 15 kets.
        dict(name="modes_ff", family="modes", d1=199, d2=3, d3=201, kets=15, form="ff"),
        # Split-operator particle Hamiltonian on a 4096-point grid, 64 wave functions.
        dict(name="particle4096_kets64", family="particle", nx=4096, ny=1, kets=64, form="c128"),
        # 256 uneven two-mode cavity models in one batched call (a parameter sweep).
        dict(name="cavities256", family="cavities", models=256, lo=8, hi=64, form="c128"),
        # Time evolution: 100 RK4 steps of a 12-spin chain.
        dict(name="rk4_chain12", family="rk4", spins=12, steps=100, form="c128"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    family = rng.choice(("jc", "chain", "chain", "lindblad", "sparse", "rows", "dense", "modes", "particle",
                         "cavities", "rk4"))
    form = rng.choice(FORMS)
    if family == "jc":
        n1, n2 = _log_int(rng, 3, 63), _log_int(rng, 3, 63)
        return dict(family=family, n1=n1, n2=n2, kets=_log_int(rng, 1, 64), form=form)
    if family == "chain":
        spins = rng.randint(8, 20)
        return dict(family=family, spins=spins, kets=_log_int(rng, 1, max(1, min(200, (1 << 22) >> spins))), form=form)
    if family == "lindblad":
        return dict(family=family, spins=rng.randint(4, 10), form=rng.choice(("c128", "c64")))
    if family == "sparse":
        n1, n2 = _log_int(rng, 7, 40), _log_int(rng, 7, 63)
        return dict(family=family, n1=n1, n2=n2, kets=_log_int(rng, 1, 256), form=form)
    if family == "rows":
        return dict(family=family, spins=rng.randint(5, 10), rows=_log_int(rng, 5, 1024), form=form)
    if family == "dense":
        n = _log_int(rng, 300, 4096)  # smaller ones are handled as local operators
        kets = _log_int(rng, 1, max(1, min(64, (1 << 27) // (n * n))))
        return dict(family=family, n=n, kets=kets, form=form)
    if family == "modes":
        d1, d2, d3 = _log_int(rng, 40, 220), rng.randint(1, 5), _log_int(rng, 40, 220)
        most = int(1.5e8 / (d1 * d2 * d3 * (d1 + d3)))
        return dict(family=family, d1=d1, d2=d2, d3=d3, kets=_log_int(rng, 1, max(1, min(16, most))), form=form)
    if family == "particle":
        if rng.random() < 0.3:  # two axes
            nx, ny = rng.choice((32, 64, 96, 128, 256)), rng.choice((32, 64, 100, 128, 256))
            return dict(family=family, nx=nx, ny=ny, kets=_log_int(rng, 1, 8), form=form)
        if rng.random() < 0.3:  # a grid that is not a power of two
            return dict(family=family, nx=_log_int(rng, 50, 800), ny=1, kets=_log_int(rng, 1, 32), form=form)
        return dict(family=family, nx=1 << rng.randint(6, 12), ny=1, kets=_log_int(rng, 1, 64), form=form)
    if family == "cavities":
        lo = rng.randint(3, 20)
        return dict(family=family, models=_log_int(rng, 2, 256), lo=lo, hi=rng.randint(lo, 64), form=form)
    return dict(family="rk4", spins=rng.randint(6, 14), steps=_log_int(rng, 5, 100), form=form)


# ---------------------------------------------------------------------------
# inputs


def _dtypes(case):
    return (torch.complex64, np.complex64) if case["form"] == "c64" else (torch.complex128, np.complex128)


def _arith(case):
    return "ff" if case["form"] == "ff" else None


def _device():
    return "cuda:0" if torch.cuda.is_available() else "cpu"


def _gen(seed, tag):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 1000003 + tag)
    return g


def _columns(case, rows, cols, seed, tag):
    """rows x cols, column-major, normalised columns."""
    t = torch.randn(cols, rows, dtype=torch.complex128, device=_device(), generator=_gen(seed, tag))
    t = t / torch.linalg.vector_norm(t, dim=1, keepdim=True)
    return t.to(_dtypes(case)[0]).t()


def _params(seed, tag, n, lo, hi):
    return np.random.default_rng([int(seed), tag]).uniform(lo, hi, n)


# ---------------------------------------------------------------------------
# Hamiltonians as lists of (coefficient, ((site, factor name), ...))


def _jc_terms(case, seed):
    omega, delta, g = _params(seed, 1, 3, 0.5, 2.0)
    dims = [case["n1"] + 1, 2, case["n2"] + 1]
    terms = [(omega, ((0, "n"),)), (omega, ((2, "n"),)), (delta / 2, ((1, "sz"),)),
             (g, ((0, "ad"), (1, "sm"))), (g, ((0, "a"), (1, "sp"))),
             (g, ((1, "sm"), (2, "ad"))), (g, ((1, "sp"), (2, "a")))]
    return dims, terms


def _chain_terms(case, seed):
    n = case["spins"]
    h = _params(seed, 2, n, -1.0, 1.0)
    terms = [(1.0, ((i, s), (i + 1, s))) for i in range(n - 1) for s in ("sx", "sy", "sz")]
    terms += [(h[i], ((i, "sz"),)) for i in range(n)]
    return [2] * n, terms


def _cavity_sizes(case):
    rng = np.random.default_rng([case["models"], case["lo"], case["hi"]])
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 2)) for _ in range(case["models"])]


def _cavity_terms(n1, n2, seed, k):
    w1, w2, chi, eps = _params(seed, 100 + k, 4, 0.1, 2.0)
    return [n1 + 1, n2 + 1], [(w1, ((0, "n"),)), (w2, ((1, "n"),)), (chi, ((0, "n"), (1, "n"))), (eps, ((0, "drive"),))]


_FACTORS = {"n": Q.number, "a": Q.destroy, "ad": Q.create, "sx": Q.sigmax, "sy": Q.sigmay, "sz": Q.sigmaz,
            "sp": Q.sigmap, "sm": Q.sigmam, "drive": lambda b, dt: Q.add(Q.destroy(b, dt), Q.create(b, dt))}


def _lazysum(dims, terms, npdt):
    """The LazySum of LazyTensors a program writes down for these terms."""
    spin = {s for _, fs in terms for s, name in fs if name[0] == "s"}
    bases = [Q.SpinBasis("1/2") if i in spin else Q.FockBasis(d - 1) for i, d in enumerate(dims)]
    b = Q.tensor_basis(*bases)
    factors = {}

    def factor(site, name):
        key = (name, len(bases[site]))
        if key not in factors:
            factors[key] = _FACTORS[name](bases[site], npdt)
        return factors[key]

    ops = tuple(Q.LazyTensor(b, b, tuple(s + 1 for s, _ in fs), tuple(factor(s, f) for s, f in fs)) for _, fs in terms)
    return Q.LazySum(b, b, [c for c, _ in terms], ops)


def _dense_matrix(case, seed, tag, n):
    """A dense n x n operator's entries (complex Gaussian, variance 1/n), host Fortran order."""
    t = torch.randn(n, n, dtype=torch.complex128, device=_device(), generator=_gen(seed, tag)) / math.sqrt(n)
    return t.to(_dtypes(case)[0]).cpu().numpy().T  # a view: column-major


def _grids(case):
    return [n for n in (case["nx"], case["ny"]) if n > 1]


_HALF = 20.0  # position grids run from -20 to 20


def _particle(case, npdt):
    bx = [PositionBasis(-_HALF, _HALF, n) for n in _grids(case)]
    bp = [MomentumBasis(b) for b in bx]
    X = bx[0] if len(bx) == 1 else Q.tensor_basis(*bx)
    P = bp[0] if len(bp) == 1 else Q.tensor_basis(*bp)
    kinetic = torch.zeros((), dtype=torch.float64)
    for b in bp:  # later subsystems are slower: they come first in the tensor
        p = torch.as_tensor(b.pmin + np.arange(b.N) * ((b.pmax - b.pmin) / b.N))
        kinetic = (p * p / 2).reshape([-1] + [1] * kinetic.ndim) + kinetic
    n = len(X)
    K = Q.Operator(P, P, Q.spdiagm(n, n, {0: kinetic.reshape(-1).numpy().astype(npdt)}, npdt))
    V = potentialoperator(X, (lambda x: 0.5 * x * x) if len(bx) == 1 else (lambda x, y: 0.5 * (x * x + y * y)), npdt)
    return Q.LazySum(X, X, [1.0, 1.0], (Q.LazyProduct((transform(X, P), K, transform(P, X))), V))


# ---------------------------------------------------------------------------


def prepare(case, seed):
    family, npdt = case["family"], _dtypes(case)[1]
    dt_form = "ff" if case["form"] == "ff" else npdt
    st = {"family": family, "arith": _arith(case)}
    if family == "cavities":
        sizes = _cavity_sizes(case)
        dims = [(a + 1) * (b + 1) for a, b in sizes]
        off = np.concatenate([[0], np.cumsum(dims)])
        x = _columns(case, int(off[-1]), 1, seed, 1).reshape(-1).contiguous() * math.sqrt(len(dims))
        y = _columns(case, int(off[-1]), 1, seed, 2).reshape(-1).contiguous() * math.sqrt(len(dims))
        batch = EV.Batch(npdt, arith=st["arith"])
        for k, (a, b) in enumerate(sizes):
            H = _lazysum(*_cavity_terms(a, b, seed, k), npdt)
            batch.add(H, x[off[k]:off[k + 1]], y[off[k]:off[k + 1]], 0.7 - 0.2j, 0.3)
        batch.info()  # compiles the batch
        return dict(st, batch=batch, y=y)
    if family == "dense":
        n = case["n"]
        b = Q.GenericBasis(n)
        op = Q.Operator(b, b, _dense_matrix(case, seed, 3, n))
    elif family == "modes":
        bs = [Q.GenericBasis(d) for d in (case["d1"], case["d2"], case["d3"])]
        f1, f3 = (Q.Operator(bs[i], bs[i], _dense_matrix(case, seed, 4 + i, len(bs[i]))) for i in (0, 2))
        b = Q.tensor_basis(*bs)
        op = Q.LazyTensor(b, b, (1, 3), (f1, f3), 0.3)
    elif family == "particle":
        op = _particle(case, npdt)
    elif family in ("jc", "sparse"):
        op = _lazysum(*_jc_terms(case, seed), npdt)
        if family == "sparse":
            op = Q.sparse(op)
            op = Q.Operator(op.basis_l, op.basis_r, op.data.astype(npdt))
    else:  # chain, lindblad, rows, rk4
        op = _lazysum(*_chain_terms(case, seed), npdt)
    n = len(op.basis_l)
    if family == "lindblad":
        b = op.basis_l
        J = [Q.LazyTensor(b, b, (i,), (Q.sigmam(Q.SpinBasis("1/2"), npdt),)) for i in range(1, case["spins"] + 1)]
        S = SO.lazy_liouvillian(op, J, rates=_params(seed, 5, case["spins"], 0.1, 1.0))
        compile_op(S.vectorised, L.QOB_LEFT, dt_form)
        rho, out = (Q.Operator(b, b, _columns(case, n, n, seed, k)) for k in (1, 2))
        return dict(st, S=S, x=rho, y=out)
    if family == "rows":
        left = Q.GenericBasis(case["rows"])
        compile_op(op, L.QOB_RIGHT, dt_form)
        x, y = (Q.Operator(left, op.basis_l, _columns(case, case["rows"], n, seed, k)) for k in (1, 2))
        return dict(st, op=op, x=x, y=y)
    compile_op(op, L.QOB_LEFT, dt_form)
    kets = case.get("kets", 1)
    if kets == 1:
        x, y = (Q.Ket(op.basis_l, _columns(case, n, 1, seed, k).reshape(-1).contiguous()) for k in (1, 2))
    else:  # a batch of kets: the columns of an operator
        b = Q.GenericBasis(kets)
        x, y = (Q.Operator(op.basis_l, b, _columns(case, n, kets, seed, k)) for k in (1, 2))
    return dict(st, op=op, x=x, y=y, steps=case.get("steps", 0))


_DT = 0.01  # RK4 step


def _alpha_beta(family):
    # Schroedinger and master-equation right-hand sides overwrite their result;
    # the others accumulate, with a complex and a real coefficient
    if family in ("jc", "particle"):
        return -1j, 0.0
    return (1.0, 0.0) if family == "lindblad" else (0.7 - 0.2j, 0.3)


def run(state):
    family = state["family"]
    if family == "cavities":
        state["batch"].run()
        return state["y"]
    if family == "rk4":
        EV.rk4(state["op"], state["x"], _DT, state["steps"], arith=state["arith"])
        return state["x"].data
    alpha, beta = _alpha_beta(family)
    if family == "lindblad":
        SO.mul_super(state["y"], state["S"], state["x"], alpha, beta)
    elif family == "rows":
        mul_(state["y"], state["x"], state["op"], alpha, beta, arith=state["arith"])
    else:
        mul_(state["y"], state["op"], state["x"], alpha, beta, arith=state["arith"])
    return state["y"].data


# ---------------------------------------------------------------------------
# the bytes and operations of one pass: every state read once and written once
# (and the result read, where it is accumulated into), operators read once


def _size(case):
    family = case["family"]
    if family in ("jc", "sparse"):
        return 2 * (case["n1"] + 1) * (case["n2"] + 1)
    if family == "dense":
        return case["n"]
    if family == "modes":
        return case["d1"] * case["d2"] * case["d3"]
    if family == "particle":
        return case["nx"] * case["ny"]
    if family == "cavities":
        return sum((a + 1) * (b + 1) for a, b in _cavity_sizes(case))
    return 1 << case["spins"]


def work(case):
    family, s = case["family"], 8 if case["form"] == "c64" else 16
    n = _size(case)
    cols = case.get("kets", 1)
    passes = 3 if _alpha_beta(family)[1] else 2
    op_bytes = 0
    if family == "jc":
        ops = 4 + 8 + 16  # merged diagonal, four couplings active on half the states, alpha
    elif family == "sparse":
        ops = 8 * 3 + 10
        op_bytes = 3 * n * (s + 4)
    elif family in ("chain", "rows", "rk4"):
        ops = 4 + 4 * (case["spins"] - 1) / 2 + 10
        cols = case.get("rows", cols)
    elif family == "lindblad":
        # merged diagonal, bonds on both sides active on half the states, the
        # jumps on a quarter of them
        ops = 8 + 2 * 4 * (case["spins"] - 1) / 2 + case["spins"] / 4 * 4 + 6
        cols = n
    elif family == "dense":
        ops = 8 * n + 10
        op_bytes = n * n * s
    elif family == "modes":
        ops = 8 * (case["d1"] + case["d3"]) + 10
    elif family == "particle":
        ops = 2 * 5 * sum(math.log2(v) for v in _grids(case)) + 40
    else:
        ops = 4 + 2 * 4 + 10
    if family == "rk4":
        # four applications a step; the state in and out once (it stays on the chip between)
        return {"bytes": 2 * n * s, "flops": 4 * case["steps"] * n * (ops + 12)}
    return {"bytes": passes * n * cols * s + op_bytes, "flops": n * cols * ops}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch alone


def _site_matrix(name, d):
    r = np.sqrt(np.arange(1, d))
    m = {"n": lambda: np.diag(np.arange(d)), "a": lambda: np.diag(r, 1), "ad": lambda: np.diag(r, -1),
         "drive": lambda: np.diag(r, 1) + np.diag(r, -1),
         "sx": lambda: np.array([[0, 1], [1, 0]]), "sy": lambda: np.array([[0, -1j], [1j, 0]]),
         "sz": lambda: np.diag([1, -1]), "sp": lambda: np.array([[0, 1], [0, 0]]),
         "sm": lambda: np.array([[0, 0], [1, 0]])}[name]()
    return m.astype(np.complex128)


def _apply_site(v, dims, site, m):
    """m on one site of the vectors v (vectors, dim), the first site fastest."""
    left, d = math.prod(dims[:site]), dims[site]
    w = v.reshape(-1, d, left)
    if d <= 3:
        out = torch.zeros_like(w)
        for i in range(d):
            for j in range(d):
                if m[i, j] != 0:
                    out[:, i, :] += complex(m[i, j]) * w[:, j, :]
    else:
        out = torch.matmul(torch.as_tensor(np.ascontiguousarray(m), device=v.device), w)
    return out.reshape(v.shape)


def _apply_terms(v, dims, terms, transpose=False):
    out = torch.zeros_like(v)
    for c, fs in terms:
        w = v
        for site, name in fs:
            m = _site_matrix(name, dims[site])
            w = _apply_site(w, dims, site, m.T if transpose else m)
        out += c * w
    return out


def _wide(t):
    return t.to(torch.complex128)


def exact(case, seed):
    family, dev = case["family"], _device()
    alpha, beta = _alpha_beta(family)
    if family == "cavities":
        sizes = _cavity_sizes(case)
        total = _size(case)
        x, y = (_wide(_columns(case, total, 1, seed, k).reshape(-1).contiguous() * math.sqrt(len(sizes))) for k in (1, 2))
        parts, off = [], 0
        for k, (a, b) in enumerate(sizes):
            dims, terms = _cavity_terms(a, b, seed, k)
            v = x[off:off + dims[0] * dims[1]].reshape(1, -1)
            parts.append(_apply_terms(v, dims, terms).reshape(-1))
            off += v.shape[1]
        return alpha * torch.cat(parts) + beta * y
    n = _size(case)
    if family == "lindblad":
        dims, terms = _chain_terms(case, seed)
        rho = _wide(_columns(case, n, n, seed, 1))
        eye = torch.eye(n, dtype=torch.complex128, device=dev)
        H = _apply_terms(eye, dims, terms).t()  # rows of the argument are vectors
        out = -1j * (H @ rho - rho @ H)
        for i, g in enumerate(_params(seed, 5, case["spins"], 0.1, 1.0)):
            jr = _apply_site(rho.t(), dims, i, _site_matrix("sm", 2)).t()               # J rho
            out += g * _apply_site(jr, dims, i, _site_matrix("sm", 2).conj())           # J rho Jdag
            p = np.diag([1.0, 0.0]).astype(np.complex128)                               # Jdag J
            out -= g / 2 * _apply_site(rho.t(), dims, i, p).t()
            out -= g / 2 * _apply_site(rho, dims, i, p.T)
        return out
    if family == "rows":
        dims, terms = _chain_terms(case, seed)
        x, y = (_wide(_columns(case, case["rows"], n, seed, k)) for k in (1, 2))
        return alpha * _apply_terms(x.contiguous(), dims, terms, transpose=True) + beta * y
    cols = case.get("kets", 1)
    x, y = (_wide(_columns(case, n, cols, seed, k)).t() for k in (1, 2))  # (kets, dim)
    if family == "dense":
        a = torch.as_tensor(np.ascontiguousarray(_dense_matrix(case, seed, 3, n).T), device=dev)  # its transpose
        h = x @ _wide(a)
    elif family == "modes":
        dims = [case["d1"], case["d2"], case["d3"]]
        h = 0.3 * x
        for i in (0, 2):
            h = _apply_site(h, dims, i, _dense_matrix(case, seed, 4 + i, dims[i]).astype(np.complex128))
    elif family == "particle":
        grids = _grids(case)[::-1]  # the first subsystem is the last tensor axis
        w = x.reshape([cols] + grids)
        shift, kin, pot = 1.0, 0.0, 0.0
        for axis, N in enumerate(grids):
            shape = [1] * len(grids)
            shape[axis] = N
            k = torch.arange(N, dtype=torch.float64, device=dev)
            dx = 2 * _HALF / N
            p = -math.pi / dx + k * (2 * math.pi / dx / N)
            q = -_HALF + k * dx
            shift = shift * (1.0 - 2.0 * (k % 2)).reshape(shape)
            kin = kin + (p * p / 2).reshape(shape)
            pot = pot + (q * q / 2).reshape(shape)
        axes = tuple(range(1, 1 + len(grids)))
        h = shift * torch.fft.ifftn(kin * torch.fft.fftn(shift * w, dim=axes), dim=axes) + pot * w
        h = h.reshape(cols, n)
    else:
        dims, terms = _jc_terms(case, seed) if family in ("jc", "sparse") else _chain_terms(case, seed)
        if family == "rk4":
            for _ in range(case["steps"]):
                k1 = -1j * _apply_terms(x, dims, terms)
                k2 = -1j * _apply_terms(x + _DT / 2 * k1, dims, terms)
                k3 = -1j * _apply_terms(x + _DT / 2 * k2, dims, terms)
                k4 = -1j * _apply_terms(x + _DT * k3, dims, terms)
                x = x + _DT / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            return x.reshape(-1)
        h = _apply_terms(x, dims, terms)
    out = alpha * h + beta * y
    return out.reshape(-1) if cols == 1 else out.t()

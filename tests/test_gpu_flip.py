"""The flip-form gather (k_gather_m) against the oracle, through mul_.

An operator is in the flip form when every merged group flips a fixed set of bits
of at most two runs of two-level subsystems, with one value: it runs k_gather_m
from 16384 elements on (strided vectors at every size).  Checked at the edges of
its shapes: one vector to ragged sets of 8 and 32, vectors that do not start on
32 bytes, rows of an operator, groups on the lowest bits, of one and two runs,
real and imaginary, a diagonal or none, beta 0 over NaN, real and complex.
Bounds: the project's parity bars, relative l2 < 1e-12 (ComplexF64 and
double-float) and < 1e-5 (ComplexF32).
"""
import numpy as np
import pytest

import oracle as OR
import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.hamiltonians import heisenberg_chain
from test_gpu_tiles import liouvillian_5

pytestmark = pytest.mark.gpu

AL = 0.7 - 0.2j
FORMS = (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12))


def _spins(n, terms):
    """LazySum of (factor, ((site, name), ...)) on n spins, sites from 1."""
    bs = Q.SpinBasis("1/2")
    b = Q.tensor_basis(*([bs] * n))
    mk = {"x": O.sigmax, "y": O.sigmay, "z": O.sigmaz, "+": O.sigmap, "-": O.sigmam}
    ops = tuple(O.LazyTensor(b, b, tuple(s for s, _ in fs), tuple(mk[k](bs) for _, k in fs)) for _, fs in terms)
    return O.LazySum(b, b, [f for f, _ in terms], ops)


def _ising(n):
    """Transverse field and next-nearest couplings (two runs), no merged diagonal."""
    t = [(0.3 + 0.1 * i, ((i, "x"),)) for i in range(1, n + 1)]
    return _spins(n, t + [(0.2 * i - 1, ((i, "x"), (i + 2, "x"))) for i in range(1, n - 1)])


def _ladder(n):
    """One stored entry per group (a jump's pattern), with a diagonal."""
    t = [(0.5 - 0.1 * i, ((i, "+"), (i + 1, "-"))) for i in range(1, n)]
    return _spins(n, t + [(1.0, ((i, "z"),)) for i in range(1, n + 1)])


def _uneven(n):
    """Two values in one group: not the flip form, the other kernels' result."""
    t = [(0.5, ((i, "+"), (i + 1, "-"))) for i in range(1, n)]
    return _spins(n, t + [(0.75, ((i, "-"), (i + 1, "+"))) for i in range(1, n)])


def _mixed(n):
    """Spins beside a three-level site that no flip touches."""
    bs, bg = Q.SpinBasis("1/2"), Q.GenericBasis(3)
    b = Q.tensor_basis(*([bs] * n + [bg]))
    s = (O.sigmax(bs), O.sigmax(bs))
    return O.LazySum(b, b, np.arange(1.0, n), tuple(O.LazyTensor(b, b, (i, i + 1), s) for i in range(1, n)))


MODELS = {"chain": lambda n: heisenberg_chain(n, seed=6), "ising": _ising, "ladder": _ladder, "uneven": _uneven,
          "mixed": _mixed, "liouvillian": lambda n: liouvillian_5(41)}


def _check(op, k, side, beta, seed, pad=0, offset=0):
    """mul_ of op on k kets (side "left") or k rows ("right") in every form; the
    device columns (rows) start `offset` elements into their buffer, leading
    dimension padded by `pad`."""
    import torch

    from qobgpu.mul import mul_

    n = len(op.basis_l)
    rows, cols = (n, k) if side == "left" else (k, n)
    rng = Q.Rng(seed)
    X = rng.complex_normal(rows * cols).reshape(rows, cols, order="F")
    Y = rng.complex_normal(rows * cols).reshape(rows, cols, order="F")
    bl = op.basis_l if side == "left" else Q.GenericBasis(k)
    br = Q.GenericBasis(k) if side == "left" else op.basis_r
    # kets one by one, or row vectors, through the oracle
    oy = O.Operator(bl, br, np.asfortranarray(Y if beta else np.zeros_like(Y)))
    ox = O.Operator(bl, br, np.asfortranarray(X))
    ref = OR.mul(oy, op, ox, AL, beta) if side == "left" else OR.mul(oy, ox, op, AL, beta)
    ref = np.asarray(ref.data if hasattr(ref, "data") and not isinstance(ref, np.ndarray) else ref)
    for form, tol in FORMS:
        dt = torch.complex64 if form == "c64" else torch.complex128

        def dev(a):
            buf = torch.full((cols * (rows + pad) + offset,), float("nan"), dtype=dt, device="cuda:0")
            v = buf[offset:].view(cols, rows + pad)[:, :rows].t()
            v.copy_(torch.as_tensor(a, device="cuda:0"))
            return v

        xd, yd = dev(X), dev(Y if beta else np.full_like(Y, np.nan))
        args = (op, O.Operator(bl, br, xd)) if side == "left" else (O.Operator(bl, br, xd), op)
        mul_(O.Operator(bl, br, yd), *args, AL, beta, arith="ff" if form == "ff" else None)
        err = rel_l2(yd.cpu().numpy().astype(np.complex128), ref)
        assert err < tol, (form, k, side, beta, pad, offset, err)


@pytest.mark.parametrize("model", sorted(MODELS))
def test_kets_against_oracle(model):
    n = {"liouvillian": 5, "mixed": 11}.get(model, 12)
    for k, beta in ((5, 0.3), (8, 0.0), (33, 0.3 + 0.4j), (64, 0.3)):
        if model == "liouvillian":
            k = 16 + k
        _check(MODELS[model](n), k, "left", beta, 40 + k)


@pytest.mark.parametrize("pad,offset", [(1, 0), (2, 1), (4, 2), (0, 3)])
def test_unaligned_kets(pad, offset):
    _check(heisenberg_chain(11, seed=5), 9, "left", 0.3, 71, pad, offset)
    _check(liouvillian_5(43), 17, "left", 0.0, 72, pad, offset)


@pytest.mark.parametrize("rows", [1, 3, 31, 33, 130])
@pytest.mark.parametrize("model", ["chain", "ising", "ladder", "uneven", "mixed", "liouvillian"])
def test_rows_against_oracle(model, rows):
    _check(MODELS[model](6), rows, "right", 0.3 if rows % 2 else 0.0, 90 + rows, pad=rows % 4)


def test_small_chains_one_large_batch():
    """The shortest chains: two sites (the whole index below the block) up."""
    for n in (2, 3, 4):
        _check(heisenberg_chain(n, seed=n), (1 << 14) // 2 ** n + 5, "left", 0.3, 110 + n)


def test_one_ket_at_the_threshold():
    for n in (13, 14, 15):
        _check(heisenberg_chain(n, seed=4), 1, "left", 0.3, 120 + n)


def test_factor_changes_reach_the_kernel():
    """set_factors between calls: new values, a group that vanishes and one whose
    entries stop being equal (the structure is rebuilt)."""
    H = heisenberg_chain(12, seed=9)
    f = H.factors.copy()
    for k, change in enumerate((lambda g: g * 1.5, lambda g: np.where(np.arange(len(g)) < 2, 0.0, g),
                                lambda g: np.where(np.arange(len(g)) == 3, 0.25, g), lambda g: g)):
        H.set_factors(change(f))
        _check(H, 6, "left", 0.3, 130 + k)


def test_nonfinite_inputs_stay_where_they_couple():
    """Inf at one index reaches the outputs that it couples to and no other."""
    import torch

    from qobgpu.mul import mul_

    H = _ladder(12)
    n = len(H.basis_l)
    X = Q.Rng(7).complex_normal(n * 5).reshape(n, 5, order="F")
    X[1234] = np.inf
    want = np.abs(np.asarray(O.sparse(H).data[:, [1234]].todense())).ravel() > 0
    for form, _ in FORMS:
        dt = torch.complex64 if form == "c64" else torch.complex128
        x = torch.as_tensor(np.ascontiguousarray(X.T), device="cuda:0").to(dt).t()
        y = torch.zeros(5, n, dtype=dt, device="cuda:0").t()
        b = Q.GenericBasis(5)
        mul_(O.Operator(H.basis_l, b, y), H, O.Operator(H.basis_r, b, x), AL, 0.0, arith="ff" if form == "ff" else None)
        got = ~np.isfinite(y.cpu().numpy())
        assert np.array_equal(got.any(axis=1), want), form


def test_tuner_reports_the_flip_kernel():
    import ctypes as C

    from qobgpu import _lib as L
    from qobgpu.device import get_context, handle, raise_for

    ctx, H = get_context(0), heisenberg_chain(12, seed=8)
    times, chosen = (C.c_double * 59)(), C.c_int()
    raise_for(L.lib().qob_op_tune_ex(ctx.ptr, handle(ctx, H).ptr, L.QOB_LEFT, L.QOB_C128, 64, times, 59,
                                     C.byref(chosen)), ctx)
    assert times[58] > 0
    if min(t for t in times if t > 0) == times[58]:
        assert (chosen.value >> 29) & 1
    _check(H, 64, "left", 0.3, 150)

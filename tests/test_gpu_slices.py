"""Dense operators and mode products from digit planes on the tensor cores
(k_slice.cu) against the oracle, through mul_.

The calls are large enough for that path (from 1e7 to 3e8 flops by form); the
sizes lie at its edges: rows and vectors that do not fill a tile of 64 rows or 16 /
32 vectors, contracted lengths around a k step (16) and a chunk (256), one or
several blocks to a row tile, vectors on either side of the product.  Tiles with
components that are not finite, far from 1 or 2^-40 and more below the largest run
in the form's own arithmetic.  Bounds: the project's parity bars, relative l2 <
1e-12 (ComplexF64, double-float) and < 1e-5 (ComplexF32); ComplexF64 also against
128-bit products where the sums, exact but for the last rounding of each chunk of
256, keep 4e-16.
"""
import numpy as np
import pytest

import oracle as OR
import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O

pytestmark = pytest.mark.gpu

AL = 0.7 - 0.2j
FORMS = (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12))


def _matrix(rng, m, n):
    return np.asfortranarray(rng.complex_normal(m * n).reshape(m, n, order="F") / np.sqrt(n))


def _device(a, form, pad=0):
    """Column-major device copy of a, leading dimension padded."""
    import torch

    dt = torch.complex64 if form == "c64" else torch.complex128
    buf = torch.full((a.shape[1], a.shape[0] + pad), float("nan"), dtype=dt, device="cuda:0")
    v = buf[:, :a.shape[0]].t()
    v.copy_(torch.as_tensor(a, device="cuda:0"))
    return v


def _mul(op, X, Y, form, beta, side="left", pad=0, alpha=AL):
    import ctypes as C

    from qobgpu import _lib as L
    from qobgpu.device import get_context, raise_for
    from qobgpu.mul import mul_

    xd, yd = _device(X, form, pad), _device(Y, form, pad)
    k = Q.GenericBasis(X.shape[1] if side == "left" else X.shape[0])
    arith = "ff" if form == "ff" else None
    if side == "left":
        mul_(O.Operator(op.basis_l, k, yd), op, O.Operator(op.basis_r, k, xd), alpha, beta, arith=arith)
    else:
        mul_(O.Operator(k, op.basis_r, yd), O.Operator(k, op.basis_l, xd), op, alpha, beta, arith=arith)
    got = yd.cpu().numpy().astype(np.complex128)
    flags = C.c_uint()
    raise_for(L.lib().qob_device_status(get_context(0).ptr, None, C.byref(flags)), get_context(0))
    assert flags.value == 0
    return got


def _dense(a):
    return O.Operator(Q.GenericBasis(a.shape[0]), Q.GenericBasis(a.shape[1]), a)


@pytest.mark.parametrize("m,n,k", [(300, 272, 17), (321, 511, 16), (513, 300, 33), (260, 1025, 8), (1030, 257, 64)])
@pytest.mark.parametrize("beta", [0.0, 0.3, 0.3 - 0.1j])
def test_dense_against_oracle(m, n, k, beta):
    rng = Q.Rng(m + n + k)
    a = _matrix(rng, m, n)
    X, Y = rng.kets_data(n, k), rng.kets_data(m, k)
    ref = AL * (a @ X) + beta * Y
    for form, tol in FORMS:
        got = _mul(_dense(a), X, Y if beta else np.full_like(Y, np.nan), form, beta, pad=k % 3)
        assert rel_l2(got, ref) < tol, (form, rel_l2(got, ref))


@pytest.mark.parametrize("rows", [70, 130])
def test_rows_times_dense(rows):
    rng = Q.Rng(rows)
    a = _matrix(rng, 300, 340)
    X, Y = rng.kets_data(rows, 300), rng.kets_data(rows, 340)
    ref = AL * (X @ a) + 0.3 * Y
    for form, tol in FORMS:
        assert rel_l2(_mul(_dense(a), X, Y, form, 0.3, side="right"), ref) < tol, form


@pytest.mark.parametrize("dims,sites,k", [((70, 5, 66), (1, 3), 30), ((3, 130, 65), (2, 3), 40),
                                           ((257, 2, 40), (1, 3), 60), ((66, 64), (1, 2), 200)])
@pytest.mark.parametrize("side", ["left", "right"])
def test_mode_products_against_oracle(dims, sites, k, side):
    rng = Q.Rng(sum(dims) + k)
    bs = [Q.GenericBasis(d) for d in dims]
    b = Q.tensor_basis(*bs)
    facs = tuple(O.Operator(bs[s - 1], bs[s - 1], _matrix(rng, dims[s - 1], dims[s - 1])) for s in sites)
    op = O.LazyTensor(b, b, sites, facs, 0.3)
    n = len(b)
    shape = (n, k) if side == "left" else (k, n)
    X, Y = rng.kets_data(*shape), rng.kets_data(*shape)
    kb = Q.GenericBasis(k)
    if side == "left":
        ref = OR.mul(O.Operator(b, kb, Y.copy(order="F")), op, O.Operator(b, kb, X), AL, 0.3)
    else:
        ref = OR.mul(O.Operator(kb, b, Y.copy(order="F")), O.Operator(kb, b, X), op, AL, 0.3)
    ref = np.asarray(ref)
    for form, tol in FORMS:
        got = _mul(op, X, Y, form, 0.3, side=side)
        assert rel_l2(got, ref) < tol, (form, rel_l2(got, ref))


def test_complexf64_against_128_bit_products():
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("no wider type on this machine")
    rng = Q.Rng(5)
    a, X = _matrix(rng, 260, 700), rng.kets_data(700, 24)
    got = _mul(_dense(a), X, np.zeros((260, 24), np.complex128, order="F"), "c128", 0.0, alpha=1.0)
    rows = np.arange(0, 260, 17)
    ref = a[rows].astype(np.clongdouble) @ X.astype(np.clongdouble)
    err = np.sqrt(float((abs(got[rows] - ref) ** 2).sum() / (abs(ref) ** 2).sum()))
    assert err < 4e-16, err


@pytest.mark.parametrize("form,tol", FORMS)
def test_graded_and_extreme_vectors_run_in_the_forms_arithmetic(form, tol):
    """Component by component, where one scale per vector would lose small ones."""
    rng = Q.Rng(6)
    a = _matrix(rng, 300, 300)
    a[:, :8] = 0.0
    a[:8, :8] = np.eye(8)
    a[:8, 8:] = 0.0
    X = rng.kets_data(300, 40)
    X[:8, 3] *= 2.0 ** -45   # 2^-45 below the rest of its vector
    X[:, 20] *= 2.0 ** (-60 if form == "c64" else -70)
    ref = a @ X
    got = _mul(_dense(a), X, np.zeros_like(X), form, 0.0, alpha=1.0)
    assert rel_l2(got[:8, 3], ref[:8, 3]) < tol
    if form != "ff":  # vector 20 lies below 2^-74, where double-float arithmetic keeps 24 bits
        assert rel_l2(got[:, 20], ref[:, 20]) < tol
    assert rel_l2(got, ref) < tol


@pytest.mark.parametrize("form,tol", FORMS)
def test_nonfinite_vectors_stay_in_their_column(form, tol):
    rng = Q.Rng(7)
    a, X = _matrix(rng, 300, 300), rng.kets_data(300, 70)
    X[5, 11] = np.nan
    X[9, 40] = np.inf
    got = _mul(_dense(a), X, np.zeros_like(X), form, 0.0)
    bad = ~np.isfinite(got).all(axis=0)
    assert list(np.flatnonzero(bad)) == [11, 40]
    keep = ~bad
    assert rel_l2(got[:, keep], AL * (a @ X[:, keep])) < tol


def test_graded_matrix_keeps_the_fma_kernels():
    rng = Q.Rng(8)
    a, X = _matrix(rng, 300, 300), rng.kets_data(300, 32)
    a[7, :] *= 2.0 ** (-60.0 * np.arange(300) / 300)
    a = np.asfortranarray(a)
    for form, tol in FORMS:
        assert rel_l2(_mul(_dense(a), X, np.zeros_like(X), form, 0.0), AL * (a @ X)) < tol, form


def test_recorded_product_reads_new_inputs():
    """A product recorded in a CUDA graph after a first call, replayed on new vectors."""
    import ctypes as C

    import torch
    from qobgpu import _lib as L
    from qobgpu.device import get_context, handle, raise_for

    rng = Q.Rng(9)
    a = _matrix(rng, 400, 400)
    op, lib, ctx = _dense(a), L.lib(), get_context(0)
    h = handle(ctx, op)
    x, y = _device(rng.kets_data(400, 16), "c128"), _device(np.zeros((400, 16), np.complex128), "c128")
    s = torch.cuda.Stream()
    sp = C.c_void_p(s.cuda_stream)

    def call():
        raise_for(lib.qob_mul(ctx.ptr, L.QOB_LEFT, 0, h.ptr, L.QOB_C128, 1.0, 0.0, C.c_void_p(x.data_ptr()), 400, 16, 400,
                              0.0, 0.0, C.c_void_p(y.data_ptr()), 400, 16, 400, sp), ctx)

    torch.cuda.synchronize()
    call()
    s.synchronize()
    g = C.c_void_p()
    raise_for(lib.qob_graph_begin(ctx.ptr, sp), ctx)
    call()
    raise_for(lib.qob_graph_end(ctx.ptr, sp, C.byref(g)), ctx)
    for _ in range(2):
        X = rng.kets_data(400, 16)
        x.copy_(torch.as_tensor(X))
        torch.cuda.synchronize()
        raise_for(lib.qob_graph_launch(ctx.ptr, g, sp), ctx)
        s.synchronize()
        assert rel_l2(y.cpu().numpy(), a @ X) < 1e-12
    lib.qob_graph_free(ctx.ptr, g)

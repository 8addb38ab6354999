"""FFTOperator passes over the lengths, line counts, strides and scalars where the kernels of
fft.cu take another turn, against the oracle's restated mul!.

Lengths: 8 (one stage) to 2048 with every remainder of log2 n by 3, 512 and more with few
lines (four-step) and with many (one block a line), below 8 and other lengths (direct
DFT, even and odd, few and many lines).  Bounds: the project's bars, relative l2
1e-12 (ComplexF64, double-float) and 1e-5 (ComplexF32).
"""
import numpy as np
import pytest

import oracle as OR
import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.bases import MomentumBasis, PositionBasis
from qobgpu.particle import transform

pytestmark = pytest.mark.gpu

AL, BE = 0.7 - 0.2j, 0.3 + 0.1j


def _dev(a, form):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a.T)).to(torch.complex64 if form == "c64" else torch.complex128).cuda().t()


def _check(T, cols, left, seed, scalars=((1.0, 0.0), (AL, 0.0), (1.0, 1.0), (AL, BE))):
    """T A (left) or A T on `cols` columns / rows, scalar forms and precisions."""
    from qobgpu.mul import mul_

    n, g = len(T.basis_l), Q.GenericBasis(cols)
    rng = Q.Rng(seed)
    shape = (n, cols) if left else (cols, n)
    a, y = (np.asfortranarray(rng.complex_normal(n * cols).reshape(shape, order="F")) for _ in range(2))
    bl, br = ((T.basis_l, g), (T.basis_r, g)) if left else ((g, T.basis_r), (g, T.basis_l))
    for al, be in scalars:
        A, Y = O.Operator(*br, a), O.Operator(*bl, y)
        ref = OR.mul(Y, T, A, al, be) if left else OR.mul(Y, A, T, al, be)
        for form, tol in (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12)):
            out, dA = O.Operator(*bl, _dev(y, form)), O.Operator(*br, _dev(a, form))
            mul_(out, *((T, dA) if left else (dA, T)), al, be, arith="ff" if form == "ff" else None)
            assert rel_l2(out.data.cpu().numpy().astype(np.complex128), ref) < tol, (form, al, be)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 16, 32, 64, 99, 100, 128, 512, 1024, 2048])
@pytest.mark.parametrize("cols", [1, 5, 170])
def test_lines(n, cols):
    bx = PositionBasis(-3.0, 4.0, n)
    T = transform(MomentumBasis(bx), bx) if n % 3 else transform(bx, MomentumBasis(bx))
    _check(T, cols, True, 800 + n)


@pytest.mark.parametrize("n", [8, 24, 64, 1024])
def test_rows(n):
    """Rows of an operator: elements a column apart."""
    bx = PositionBasis(-3.0, 4.0, n)
    _check(transform(MomentumBasis(bx), bx), 7, False, 900 + n)


@pytest.mark.parametrize("shape", [(8, 16), (3, 32), (64, 2), (5, 8, 7), (16, 512)])
def test_axes(shape):
    """Several axes: lines whose elements are a stride apart, neighbours side by side."""
    bxs = [PositionBasis(-3.0 - i, 4.0 + i, n) for i, n in enumerate(shape)]
    T = transform(Q.tensor_basis(*[MomentumBasis(b) for b in bxs]), Q.tensor_basis(*bxs))
    _check(T, 3, True, 950 + len(shape))


def _diag(b, rng, real):
    v = rng.complex_normal(len(b))
    return O.Operator(b, b, O.spdiagm(len(b), len(b), {0: v.real.copy() if real else v}))


@pytest.mark.parametrize("shape", [(8,), (64,), (512,), (2048,), (8, 16), (3, 32), (32, 3), (16, 8, 32), (16, 512)])
@pytest.mark.parametrize("cols", [1, 170])
@pytest.mark.parametrize("left", [True, False])
def test_transform_diagonal_transform(shape, cols, left):
    """Products T' D T: alone, in a longer chain, and beside diagonal terms of the same and
    of other coefficients; lengths with equal and unequal four-step halves, last axes with and
    without an FFT, lines that only the four-step form spreads."""
    bxs = [PositionBasis(-3.0 - i, 4.0 + i, n) for i, n in enumerate(shape)]
    X = bxs[0] if len(bxs) == 1 else Q.tensor_basis(*bxs)
    cols = min(cols, 2**18 // len(X))  # the oracle's time
    P = MomentumBasis(X) if len(bxs) == 1 else Q.tensor_basis(*[MomentumBasis(b) for b in bxs])
    rng = Q.Rng(970 + len(X) + cols)
    real = cols == 1
    T, Ti, D, V = transform(P, X), transform(X, P), _diag(P, rng, real), _diag(X, rng, not real)
    prod = O.LazyProduct((Ti, D, T))
    _check(prod, cols, left, 1, scalars=((AL, BE),))
    _check(O.LazyProduct((V, Ti, D, T)), cols, left, 2, scalars=((1.0, 0.0),))
    for cs in ([1.0, 1.0], [0.5, 2.0 - 1j]):
        _check(O.LazySum(X, X, cs, (prod, V)), cols, left, 3, scalars=((-1j, 0.0), (AL, BE)))

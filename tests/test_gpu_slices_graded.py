"""Dense operators and mode products on graded data: vectors and matrices whose
components differ by many powers of two (Fock tails, wave packets, thermal states,
displacement rows), where one scale per row and vector does not hold every
component.  Through mul_, in the three forms, at sizes that run from digit planes
(k_slice.cu) when the components are of about one size.

Tolerances.  A product of one nonzero pair is exact in ComplexF64 and ComplexF32
and holds 48 bits in double-float: 2^-52, 2^-23, 2^-46 leave one unit of rounding.
Sums: the classical bound of a chain of multiply-adds, component by component,
|error| <= 2 n u sum_k |a_ik| |x_k| with u = 2^-53, 2^-24, 2^-46 (a double-float
product keeps 46 bits), beside the project's bars of relative l2 < 1e-12 (ComplexF64,
double-float) and < 1e-5 (ComplexF32).
"""
import numpy as np
import pytest

import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from test_gpu_slices import _dense, _matrix, _mul

pytestmark = pytest.mark.gpu

FORMS = (("c128", 1e-12, 2.0 ** -52, 2.0 ** -53), ("c64", 1e-5, 2.0 ** -23, 2.0 ** -24),
         ("ff", 1e-12, 2.0 ** -46, 2.0 ** -46))
SHIFTS = (2, 5, 8, 10, 14, 20, 26, 30, 32, 35, 39, 41, 45)


def _rounded(a, form):
    """What the form is given: ComplexF32 data are compared as they are stored."""
    return a.astype(np.complex64).astype(np.complex128) if form == "c64" else a


def _product(a, X, form):
    op = a if isinstance(a, O.Operator) else _dense(a)
    return _mul(op, X, np.zeros((len(op.basis_l), X.shape[1]), np.complex128, order="F"), form, 0.0, alpha=1.0)


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
@pytest.mark.parametrize("n", [300, 1025])
def test_identity_rows_on_small_components(n, form, tol, unit, u):
    rng = Q.Rng(n)
    a = _matrix(rng, n, n)
    a[:8, :] = 0.0
    a[:8, :8] = np.eye(8)
    a, X0 = _rounded(a, form), rng.kets_data(n, 33)
    op, worst = _dense(a), {}
    for e in SHIFTS:  # a call each: a vector left to the other kernels takes its neighbours with it
        X = X0.copy(order="F")
        X[:8, 3:9] *= 2.0 ** -e
        X = _rounded(X, form)
        got = _product(op, X, form)
        worst[e] = float((abs(got[:8] - X[:8]) / abs(X[:8])).max())
        assert rel_l2(got, a @ X) < tol, e
    assert max(worst.values()) < unit, worst


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
def test_identity_on_small_components(form, tol, unit, u):
    """Every row of the matrix holds one component exactly."""
    X0 = Q.Rng(1).kets_data(320, 40)
    op, worst = _dense(np.asfortranarray(np.eye(320, dtype=np.complex128))), {}
    for e in SHIFTS:
        X = X0.copy(order="F")
        X[7:] *= 2.0 ** -e
        X = _rounded(X, form)
        got = _product(op, X, form)
        worst[e] = float((abs(got - X) / abs(X)).max())
    assert max(worst.values()) < unit, worst


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
def test_basis_kets_return_graded_columns(form, tol, unit, u):
    rng = Q.Rng(2)
    n = 320
    a = _matrix(rng, n, n) * 2.0 ** -np.array([SHIFTS[j % len(SHIFTS)] if j % 3 else 0 for j in range(n)])[None, :]
    a = _rounded(np.asfortranarray(a), form)
    X = np.zeros((n, 64), np.complex128, order="F")
    X[5 * np.arange(64), np.arange(64)] = 1.0
    got = _product(a, X, form)
    ref = a[:, 5 * np.arange(64)]
    assert float((abs(got - ref) / abs(ref)).max()) < unit


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
@pytest.mark.parametrize("bits", [10, 20, 30, 40])
@pytest.mark.parametrize("n", [256, 600])
def test_opposite_gradings(n, bits, form, tol, unit, u):
    """Matrix falling and vectors rising along the contracted index: every term of a
    sum has the same size.  The vectors alone, and the matrix alone, too."""
    rng = Q.Rng(bits + n)
    g = 2.0 ** (-bits * (np.arange(n) % 256) / 255.0)
    a, X = _matrix(rng, 300, n), rng.kets_data(n, 40)
    for fa, fx in ((g, 1 / g), (np.ones(n), g), (g, np.ones(n))):
        am, Xm = _rounded(np.asfortranarray(a * fa[None, :]), form), _rounded(np.asfortranarray(X * fx[:, None]), form)
        got, ref = _product(am, Xm, form), am @ Xm
        assert rel_l2(got, ref) < tol
        # the reference's own rounding is of the ComplexF64 bound's size
        assert (abs(got - ref) <= 2 * n * (u + 2.0 ** -53) * (abs(am) @ abs(Xm))).all()


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
def test_real_parts_far_below_imaginary_ones(form, tol, unit, u):
    """Re and Im of a result are sums of their own: small real parts keep their bits."""
    rng = Q.Rng(3)
    a = _rounded(np.asfortranarray(_matrix(rng, 300, 300).real.astype(np.complex128)), form)
    X = rng.kets_data(300, 40)
    X = _rounded(np.asfortranarray(X.real * 2.0 ** -33 + 1j * X.imag), form)
    got, ref = _product(a, X, form), a @ X
    assert rel_l2(got.real, ref.real) < tol and rel_l2(got.imag, ref.imag) < tol


def _coherent(n, alphas):
    k = np.arange(n)
    lg = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, n)))])
    return np.asfortranarray(np.stack([np.exp(-abs(z) ** 2 / 2 + k * np.log(abs(z)) - lg / 2) * np.exp(1j * k * np.angle(z))
                                       for z in alphas], axis=1))


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
@pytest.mark.parametrize("n", [300, 1000])
def test_coherent_states_and_wave_packets(n, form, tol, unit, u):
    rng = Q.Rng(4)
    al = 1 + 0.2 * np.arange(32)
    x = np.linspace(-12, 12, n)
    packets = np.exp(-(x[:, None] - 4 * np.sin(np.arange(32.0)[None, :])) ** 2 / 2 + 2j * x[:, None])
    for X in (_coherent(n, al * np.exp(1j * al)), packets / np.linalg.norm(packets, axis=0)):
        X = np.asfortranarray(np.where(abs(X) > 1e-30, X, 0))  # within every form's range
        a, X = _rounded(_matrix(rng, n, n), form), _rounded(X, form)
        got, ref = _product(a, X, form), a @ X
        assert rel_l2(got, ref) < tol
        assert (abs(got - ref) <= 2 * n * (u + 2.0 ** -53) * (abs(a) @ abs(X)) + 1e-36).all()


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
@pytest.mark.parametrize("side", ["left", "right"])
def test_graded_mode_products(side, form, tol, unit, u):
    rng = Q.Rng(5)
    dims, k = (66, 3, 70), 60
    bs = [Q.GenericBasis(d) for d in dims]
    b = Q.tensor_basis(*bs)
    f = [np.asfortranarray(_rounded(_matrix(rng, d, d), form)) for d in (66, 70)]
    f[0][:4, :] = np.eye(4, 66)
    op = O.LazyTensor(b, b, (1, 3), (O.Operator(bs[0], bs[0], f[0]), O.Operator(bs[2], bs[2], f[1])))
    x0 = rng.kets_data(len(b), k).reshape(66, 3, 70, k, order="F")
    A, B = (f[0], f[1]) if side == "left" else (f[0].T, f[1].T)
    for e in SHIFTS:
        x = x0.copy(order="F")
        x[:4] *= 2.0 ** -e
        x = _rounded(x, form)
        X = np.asfortranarray(x.reshape(len(b), k, order="F"))
        ref = np.tensordot(np.tensordot(A, x, (1, 0)), B, (2, 1)).transpose(0, 1, 3, 2)  # (a, s, b, ket)
        if side == "left":
            got = _mul(op, X, np.zeros_like(X), form, 0.0, alpha=1.0)
        else:
            got = _mul(op, np.asfortranarray(X.T), np.zeros((k, len(b)), np.complex128, order="F"), form, 0.0,
                       side="right", alpha=1.0).T
        got = got.reshape(66, 3, 70, k, order="F")
        assert rel_l2(got, ref) < tol, e
        if side == "left":  # rows 0 .. 3 of the first factor are the identity's
            assert rel_l2(got[:4], ref[:4]) < tol, e


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
@pytest.mark.parametrize("side", ["left", "right"])
def test_graded_kets_among_others(side, form, tol, unit, u):
    """Some tiles of vectors from digits and some not, into a result that is accumulated."""
    rng = Q.Rng(6)
    n, k = 66 * 3 * 70, 60
    bs = [Q.GenericBasis(d) for d in (66, 3, 70)]
    b = Q.tensor_basis(*bs)
    f = [_rounded(_matrix(rng, d, d), form) for d in (66, 70)]
    modes = O.LazyTensor(b, b, (1, 3), (O.Operator(bs[0], bs[0], f[0]), O.Operator(bs[2], bs[2], f[1])))
    A, B = (f[0], f[1]) if side == "left" else (f[0].T, f[1].T)
    a = _rounded(_matrix(rng, 330, 330), form)
    for op, dim, ref in (
            (modes, n, lambda v: np.tensordot(np.tensordot(A, v.reshape(66, 3, 70, -1, order="F"), (1, 0)), B,
                                              (2, 1)).transpose(0, 1, 3, 2).reshape(n, -1, order="F")),
            (_dense(a), 330, lambda v: (a if side == "left" else a.T) @ v)):
        cols = k if op is modes else 150
        X, Y = rng.kets_data(dim, cols), rng.kets_data(dim, cols)
        for c in (1, 40, cols - 1):
            X[:, c] *= 2.0 ** -(30.0 * np.arange(dim) / dim)
            X[::7, c] = 0.0
        X, Y = _rounded(X, form), _rounded(Y, form)
        want = (0.7 - 0.2j) * ref(X) + (0.3 - 0.1j) * Y
        if side == "left":
            got = _mul(op, X, Y, form, 0.3 - 0.1j)
        else:
            got = _mul(op, np.asfortranarray(X.T), np.asfortranarray(Y.T), form, 0.3 - 0.1j, side="right").T
        assert rel_l2(got, want) < tol
        for c in (0, 1, 40, cols - 1):
            assert rel_l2(got[:, c], want[:, c]) < tol, c


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
def test_graded_kets_cost_what_the_fma_kernels_do(form, tol, unit, u):
    """The same kets under a matrix that has no planes (a graded one) go to the FMA kernels at once."""
    import torch

    from qobgpu.mul import mul_

    n, k = 2048, 16
    g = torch.Generator(device="cuda:0")
    g.manual_seed(7)
    dt = torch.complex64 if form == "c64" else torch.complex128
    a = (torch.randn(n, n, dtype=torch.complex128, device="cuda:0", generator=g) / 45).to(dt).cpu().numpy().T
    x = torch.randn(k, n, dtype=torch.complex128, device="cuda:0", generator=g)
    x[:, 100:] *= 2.0 ** -30
    y = torch.zeros(k, n, dtype=dt, device="cuda:0").t()
    b, bk = Q.GenericBasis(n), Q.GenericBasis(k)
    X, Y = O.Operator(b, bk, x.to(dt).t()), O.Operator(b, bk, y)
    graded = np.asfortranarray(a.copy())
    graded[0] *= (2.0 ** -(30.0 * np.arange(n) / n)).astype(a.real.dtype)
    ms = []
    for m in (a, graded):
        op, best = O.Operator(b, b, m), np.inf
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(4):
                mul_(Y, op, X, arith="ff" if form == "ff" else None)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]) / 4)
        ms.append(best)
    # three launches that find nothing to do beside kernels of 50 us and more
    assert ms[0] < 2 * ms[1], ms


@pytest.mark.parametrize("form,tol,unit,u", FORMS)
def test_more_vectors_than_one_fma_launch(form, tol, unit, u):
    """The gate of the second launch, of one vector: graded (left to it) and not."""
    import torch

    from qobgpu.mul import mul_

    n, k = 300, (4 if form == "ff" else 8) * 65535 + 1
    a = _rounded(_matrix(Q.Rng(8), n, n), form)
    dt = torch.complex64 if form == "c64" else torch.complex128
    g = torch.Generator(device="cuda:0")
    g.manual_seed(9)
    x = torch.randn(k, n, dtype=torch.complex64, device="cuda:0", generator=g).to(dt)
    y0 = torch.randn(k, n, dtype=torch.complex64, device="cuda:0", generator=g).to(dt)
    b, bk, op = Q.GenericBasis(n), Q.GenericBasis(k), _dense(a)
    for graded in (False, True):
        if graded:
            x[-1, 10:] *= 2.0 ** -30
        y = y0.clone()
        mul_(O.Operator(b, bk, y.t()), op, O.Operator(b, bk, x.t()), 0.7, 0.3, arith="ff" if form == "ff" else None)
        for c in (0, 40000, k - 40, k - 2, k - 1):
            want = 0.7 * (a @ x[c].cpu().numpy().astype(np.complex128)) + 0.3 * y0[c].cpu().numpy().astype(np.complex128)
            assert rel_l2(y[c].cpu().numpy().astype(np.complex128), want) < tol, (graded, c)

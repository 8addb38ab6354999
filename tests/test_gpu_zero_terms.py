"""Operators whose terms hold no entry (a factor of zeros): the result is beta times itself,
alone, in a LazyProduct and in RK4, in every form; beta = 0 over NaN."""
import numpy as np
import pytest

import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.evolution import rk4
from test_gpu_slices import _device

pytestmark = pytest.mark.gpu

FORMS = (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12))


def _zero(b, sparse):
    n = len(b)
    return O.Operator(b, b, O.spdiagm(n, n, {}) if sparse else np.zeros((n, n), np.complex128, order="F"))


def _models():
    bs = Q.SpinBasis("1/2")
    b = Q.tensor_basis(bs, bs, bs)
    sx, sz = O.sigmax(bs), O.sigmaz(bs)
    for sparse in (True, False):
        z = _zero(bs, sparse)
        none = O.LazyTensor(b, b, (1, 2), (z, sx))
        yield none
        yield O.LazySum(b, b, [0.3 - 0.2j, 1.0], (none, none))
        yield O.LazyProduct((O.LazyTensor(b, b, (3,), (sx,)), none))
        yield O.LazySum(b, b, [0.5, 1.0, 2.0], (O.LazyProduct((none, O.LazyTensor(b, b, (2,), (sz,)))), none,
                                                 O.LazyTensor(b, b, (1, 3), (sx, sz))))


@pytest.mark.parametrize("form,tol", FORMS)
@pytest.mark.parametrize("model", range(8))
def test_terms_without_entries(model, form, tol):
    from qobgpu.mul import mul_

    op = list(_models())[model]
    m, b = np.asarray(O.dense(op).data), op.basis_l
    rng = Q.Rng(model)
    X, Y = rng.kets_data(8, 5), rng.kets_data(8, 5)
    kb = Q.GenericBasis(5)
    for beta in (0.0, 0.3 - 0.1j):
        x, y = _device(X, form), _device(Y if beta else np.full_like(Y, np.nan), form)
        mul_(O.Operator(b, kb, y), op, O.Operator(b, kb, x), 0.7 - 0.2j, beta, arith="ff" if form == "ff" else None)
        want, got = (0.7 - 0.2j) * (m @ X) + beta * Y, y.cpu().numpy()
        assert rel_l2(got, want) < tol if np.any(want) else not np.any(got)
    psi = _device(X[:, :1] / np.linalg.norm(X[:, 0]), form).reshape(-1).contiguous()
    v = psi.cpu().numpy().astype(np.complex128)
    rk4(op, psi, 1e-2, 3, arith="ff" if form == "ff" else None)
    for _ in range(3):
        k1 = -1j * (m @ v)
        k2 = -1j * (m @ (v + 5e-3 * k1))
        k3 = -1j * (m @ (v + 5e-3 * k2))
        k4 = -1j * (m @ (v + 1e-2 * k3))
        v = v + 1e-2 / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    assert rel_l2(psi.cpu().numpy(), v) < tol

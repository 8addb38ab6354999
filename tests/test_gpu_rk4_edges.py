"""The one-launch RK4 (rk4.cu) at the edges of its launches: more steps than one launch makes
(1024), lists at the sizes where resident blocks run out (2^16 and 2^17 entries),
rows too wide for lists up to the largest state that walks the tables (2^16), and the size above,
which takes four launches a step.  The kernels hold the batched stages' arithmetic, so a long
evolution equals the same one in shorter calls to the bit; the large states are checked against
RK4 in NumPy on the sparse operator (bars as in test_gpu_rk4_grid.py: relative l2 < 1e-12 and
< 1e-5 in ComplexF32)."""
import numpy as np
import pytest

import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.evolution import rk4
from qobgpu.hamiltonians import heisenberg_chain
from test_gpu_rk4_grid import _wide

pytestmark = pytest.mark.gpu

FORMS = (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12))


def _run(H, psi0, dt, steps, form):
    import torch

    psi = torch.as_tensor(psi0, device="cuda:0").to(torch.complex64 if form == "c64" else torch.complex128)
    for n in steps:
        rk4(H, psi, dt, n, arith="ff" if form == "ff" else None)
    return psi.cpu().numpy()


@pytest.mark.parametrize("form,tol", FORMS)
@pytest.mark.parametrize("model", ["spins", "wide"])
@pytest.mark.parametrize("steps", [1025, 2049])
def test_more_steps_than_one_launch(steps, model, form, tol):
    H = heisenberg_chain(6, seed=3) if model == "spins" else _wide(17)
    psi0 = Q.Rng(21).ket_data(len(H.basis_l))
    whole = _run(H, psi0, 1e-3, (steps,), form)
    assert np.array_equal(whole, _run(H, psi0, 1e-3, (1000, 20, steps - 1020), form))
    assert abs(np.linalg.norm(whole) - 1) < 100 * tol  # a unitary evolution


def _wide_large(n):
    """66 entries a row, more than a list holds: hops of up to 33 sites."""
    b = Q.GenericBasis(n)
    d = {}
    for k in range(1, 34):
        v = 0.1 / k * np.ones(n - k)
        d[k], d[-k] = v, v
    return O.Operator(b, b, O.spdiagm(n, n, d))


@pytest.mark.parametrize("form,tol", FORMS)
@pytest.mark.parametrize("model", ["spins16", "spins17", "spins18", "hops40000", "hops65536"])
def test_large_states(model, form, tol):
    H = heisenberg_chain(int(model[5:]), seed=3) if model[0] == "s" else _wide_large(int(model[4:]))
    psi0, dt = Q.Rng(22).ket_data(len(H.basis_l)), 2e-3
    m = Q.sparse(H).data.tocsr()
    v = psi0.copy()
    for _ in range(2):
        k1 = -1j * (m @ v)
        k2 = -1j * (m @ (v + dt / 2 * k1))
        k3 = -1j * (m @ (v + dt / 2 * k2))
        k4 = -1j * (m @ (v + dt * k3))
        v = v + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    assert rel_l2(_run(H, psi0, dt, (2,), form).astype(np.complex128), v) < tol

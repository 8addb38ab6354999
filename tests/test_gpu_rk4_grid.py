"""RK4 of one state in one cooperative launch (rk4.cu) against RK4 on the host with
the oracle as right-hand side, through rk4.

Sizes: below one block of 128, a block and one more, several blocks with a ragged
last one, more entries than lists take (the table-walking kernel), rows of one and of several
stored entries, complex values, no diagonal; step counts 2 (the smallest run in
one launch) and 7.  Bounds: the project's bars for short evolutions, relative l2 <
1e-12 (ComplexF64, double-float) and < 1e-5 (ComplexF32).
"""
import numpy as np
import pytest

import oracle as OR
import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.hamiltonians import heisenberg_chain, jaynes_cummings, two_mode_cavity
from test_gpu_tiles import complex_chain

pytestmark = pytest.mark.gpu


def _hop(n):
    """Off-diagonal only, odd size."""
    b = Q.GenericBasis(n)
    return O.Operator(b, b, O.spdiagm(n, n, {1: np.linspace(0.2, 1, n - 1), -1: np.linspace(0.2, 1, n - 1)}))


def _wide(n):
    """A dense 12 x 12 factor: rows too wide for fixed-width slots."""
    bs = [Q.GenericBasis(12), Q.GenericBasis(n)]
    a = Q.Rng(3).complex_normal(144).reshape(12, 12, order="F")
    b = Q.tensor_basis(*bs)
    return O.LazyTensor(b, b, (1,), (O.Operator(bs[0], bs[0], np.asfortranarray((a + a.conj().T) / 8)),))


MODELS = {"spins6": lambda: heisenberg_chain(6, seed=3), "spins7": lambda: heisenberg_chain(7, seed=3),
          "cavity": lambda: two_mode_cavity(12, 9, seed=4), "jc": lambda: jaynes_cummings(7, 8, seed=5),
          "hop129": lambda: _hop(129), "hop1001": lambda: _hop(1001), "complex": lambda: complex_chain(8, 6),
          "wide": lambda: _wide(17), "spins13": lambda: heisenberg_chain(13, seed=3)}


@pytest.mark.parametrize("model", sorted(MODELS))
@pytest.mark.parametrize("steps", [2, 7])
def test_rk4_in_one_launch(model, steps):
    import ctypes as C

    import torch
    from qobgpu import _lib as L
    from qobgpu.device import get_context, raise_for
    from qobgpu.evolution import rk4

    H, dt = MODELS[model](), 2e-3
    n = len(H.basis_l)
    psi0 = Q.Rng(17).ket_data(n)

    def rhs(v):
        return np.asarray(OR.mul(Q.Ket(H.basis_l, np.zeros(n, np.complex128)), H, Q.Ket(H.basis_r, v), -1j, 0.0))

    ref = psi0.copy()
    for _ in range(steps):
        k1 = rhs(ref)
        k2 = rhs(ref + dt / 2 * k1)
        k3 = rhs(ref + dt / 2 * k2)
        k4 = rhs(ref + dt * k3)
        ref = ref + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    for form, tol in (("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12)):
        dt_ = torch.complex64 if form == "c64" else torch.complex128
        psi = torch.as_tensor(psi0, device="cuda:0").to(dt_)
        rk4(H, psi, dt, steps, arith="ff" if form == "ff" else None)
        assert rel_l2(psi.cpu().numpy().astype(np.complex128), ref) < tol, form
        flags = C.c_uint()
        raise_for(L.lib().qob_device_status(get_context(0).ptr, None, C.byref(flags)), get_context(0))
        assert flags.value == 0

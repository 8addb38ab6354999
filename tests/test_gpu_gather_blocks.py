"""Block sizes of the one-index gather: 64, 128 and 256 threads by how many blocks a call has
(k_gather.cuh, launch_j), over index and vector counts around those lines, against the
oracle.  Bounds: the project's bars, relative l2 1e-12 (ComplexF64) and 1e-5 (ComplexF32).
"""
import numpy as np
import pytest

import oracle as OR
import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from qobgpu.hamiltonians import two_mode_cavity
from qobgpu.mul import mul_, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,cols", [(6, 8, 1), (6, 8, 9), (40, 49, 40), (40, 49, 300), (40, 49, 620), (63, 63, 700)])
def test_block_sizes(n1, n2, cols):
    H = two_mode_cavity(n1, n2, seed=6)
    b, g, rng = H.basis_l, Q.GenericBasis(cols), Q.Rng(60 + cols)
    n = len(b)
    x, y = (O.Operator(b, g, np.asfortranarray(rng.complex_normal(n * cols).reshape(n, cols, order="F"))) for _ in range(2))
    al, be = 0.7 - 0.2j, 0.3
    ref = OR.mul(y, H, x, al, be)
    for dt, tol in ((np.complex128, 1e-12), (np.complex64, 1e-5)):
        out = to_device(y, dtype=dt)
        mul_(out, H, to_device(x, dtype=dt), al, be)
        assert rel_l2(out.data.cpu().numpy().astype(np.complex128), ref) < tol

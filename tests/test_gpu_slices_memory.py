"""Memory of the digit planes (k_slice.cu): none for an operator that meets single kets only,
made by the first call that takes them, and a call whose planes find no room runs
on the FMA kernels.  The last is injected on the host: the bounds-checked build refuses
to let a workspace slot grow beyond a limit, as an allocation would without memory."""
import os
import subprocess
import sys

import numpy as np
import pytest

import qobgpu as Q
from helpers import rel_l2
from qobgpu import operators as O
from test_gpu_slices import _dense, _device, _matrix, _mul

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_planes_for_single_kets():
    import torch

    from qobgpu import _lib as L
    from qobgpu.device import prepare
    from qobgpu.mul import mul_

    n = 2048  # 64 MB in ComplexF64
    rng = np.random.default_rng(1)
    a = np.asfortranarray(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    kets = {k: (_device(rng.standard_normal((n, k)) + 0j, "c128"), _device(np.zeros((n, k)), "c128")) for k in (1, 16)}
    _mul(_dense(a[:300, :300]), rng.standard_normal((300, 16)) + 0j, np.zeros((300, 16), np.complex128), "c128", 0.0)
    b = Q.GenericBasis(n)
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info(0)[0]]
    op = O.Operator(b, b, a)
    prepare(op, L.QOB_LEFT, np.complex128)
    for k in (1, 16):
        x, y = kets[k]
        mul_(O.Operator(b, Q.GenericBasis(k), y), op, O.Operator(b, Q.GenericBasis(k), x))
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info(0)[0])
        assert rel_l2(y.cpu().numpy(), a @ x.cpu().numpy()) < 1e-12
    matrix = n * n * 16
    assert free[0] - free[1] < 1.5 * matrix  # the matrix and the partial sums of a one-ket product
    assert free[1] - free[2] > 0.9 * matrix  # its planes


CHILD = r'''
import ctypes as C, sys
import numpy as np
sys.path[:0] = [{root!r}, {root!r} + "/quantumopticsbase.jl_gb300", {root!r} + "/oracle", {root!r} + "/tests"]
import qobgpu as Q
from qobgpu import _lib as L
from qobgpu import operators as O
from qobgpu.device import get_context, raise_for
from helpers import rel_l2
from test_gpu_slices import FORMS, _dense, _matrix, _mul
lib = L.lib()
assert L.LIB_PATH.endswith("libqobgpu_debug.so"), L.LIB_PATH
lib.qob_debug_limit_workspace.argtypes = [C.c_void_p, C.c_size_t]
ctx = get_context(0)
rng = Q.Rng(1)
bs = [Q.GenericBasis(d) for d in (66, 3, 70)]
b = Q.tensor_basis(*bs)
f = [_matrix(rng, d, d) for d in (66, 70)]
k = 60
for form, tol in FORMS:
    # a step's result (and, in double-float, its split input) fit, the planes of 12600 vectors of 70 do not
    esz = 8 if form == "c64" else 16
    raise_for(lib.qob_debug_limit_workspace(ctx.ptr, len(b) * k * esz), ctx)
    op = O.LazyTensor(b, b, (1, 3), (O.Operator(bs[0], bs[0], f[0]), O.Operator(bs[2], bs[2], f[1])))
    X, Y = rng.kets_data(len(b), k), rng.kets_data(len(b), k)
    want = 0.3 * Y + (0.7 - 0.2j) * np.tensordot(np.tensordot(f[0], X.reshape(66, 3, 70, k, order="F"), (1, 0)), f[1], (2, 1)
                                                 ).transpose(0, 1, 3, 2).reshape(len(b), k, order="F")
    assert rel_l2(_mul(op, X, Y, form, 0.3), want) < tol, form
    # with room again, a dense operator
    n = 400
    a, X, Y = _matrix(rng, n, n), rng.kets_data(n, 64), rng.kets_data(n, 64)
    raise_for(lib.qob_debug_limit_workspace(ctx.ptr, 0), ctx)
    assert rel_l2(_mul(_dense(a), X, Y, form, 0.3), 0.3 * Y + (0.7 - 0.2j) * (a @ X)) < tol, form
print("limits ok")
'''


def test_planes_without_room_leave_the_call_to_the_fma_kernels():
    sys.path.insert(0, os.path.join(ROOT, "quantumopticsbase.jl_gb300"))
    import build as qob_build

    env = dict(os.environ, QOB_LIBRARY=qob_build.build(debug_bounds=True))
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "limits ok" in r.stdout

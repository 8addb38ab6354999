"""The bounds-checked build on the kernels that test_gpu_debug_bounds.py does not reach:
the flip-form gather (k_gather_m; 16 kets of a 10-spin operator, and operator rows) and the
one-launch RK4 (k_rk4_list).  As there: one stored entry's input offset, and its group's
flip, moved past the end of the vectors, inside the same allocation; the status
reports it, an intact operator matches the oracle with a clean status."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import ctypes as C, sys
import numpy as np
sys.path[:0] = [{root!r}, {root!r} + "/quantumopticsbase.jl_gb300", {root!r} + "/oracle", {root!r} + "/tests"]
import torch
import oracle as OR
import qobgpu as Q
from qobgpu import _lib as L
from qobgpu.device import get_context, handle, raise_for
from qobgpu.hamiltonians import heisenberg_chain
from helpers import rel_l2
from test_gpu_flip import _spins
lib = L.lib()
assert L.LIB_PATH.endswith("libqobgpu_debug.so"), L.LIB_PATH
lib.qob_debug_shift_slot.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int]
ctx = get_context(0)
AL, BE, N, K = 0.7 - 0.2j, 0.3, 1024, 16
FORMS = ((L.QOB_C128, torch.complex128, 1e-12), (L.QOB_C64, torch.complex64, 1e-5), (L.QOB_C128X, torch.complex128, 1e-12))

def status():
    flags = C.c_uint()
    rc = lib.qob_device_status(ctx.ptr, None, C.byref(flags))
    return rc, flags.value, lib.qob_last_error(ctx.ptr)

def apply(H, side, form, dt):
    """y = AL H x + BE y on K kets, or on K rows, in buffers with as much room again behind them."""
    hd, rng = handle(ctx, H), Q.Rng(5)
    X, Y = rng.kets_data(N, K), rng.kets_data(N, K)
    if side == L.QOB_LEFT:
        xb, yb = (torch.zeros(2 * K, N, dtype=dt, device="cuda:0") for _ in range(2))
        xv, yv, shape = xb[:K].t(), yb[:K].t(), (N, K, N)
    else:  # K x N, column-major: a row's elements lie K apart
        xb, yb = (torch.zeros(2 * N, K, dtype=dt, device="cuda:0") for _ in range(2))
        xv, yv, shape = xb[:N], yb[:N], (K, N, K)
    xv.copy_(torch.as_tensor(X, device="cuda:0"))
    yv.copy_(torch.as_tensor(Y, device="cuda:0"))
    raise_for(lib.qob_mul(ctx.ptr, side, 0, hd.ptr, form, AL.real, AL.imag, C.c_void_p(xb.data_ptr()), *shape, BE, 0.0,
                          C.c_void_p(yb.data_ptr()), *shape, None), ctx)
    torch.cuda.synchronize()
    m = OR_dense(H) if side == L.QOB_LEFT else OR_dense(H).T
    return rel_l2(yv.cpu().numpy(), AL * (m @ X) + BE * Y)

def evolve(H, side, form, dt):
    hd, psi0 = handle(ctx, H), Q.Rng(6).ket_data(N)
    psi = torch.zeros(2 * N, dtype=dt, device="cuda:0")
    psi[:N].copy_(torch.as_tensor(psi0, device="cuda:0"))
    raise_for(lib.qob_rk4(ctx.ptr, hd.ptr, form, C.c_void_p(psi.data_ptr()), N, 1e-3, 3, 0, None), ctx)
    m, v = OR_dense(H), psi0.copy()
    for _ in range(3):
        k1 = -1j * (m @ v); k2 = -1j * (m @ (v + 5e-4 * k1)); k3 = -1j * (m @ (v + 5e-4 * k2)); k4 = -1j * (m @ (v + 1e-3 * k3))
        v = v + 1e-3 / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return rel_l2(psi[:N].cpu().numpy(), v)

def OR_dense(H):
    return np.asarray(Q.sparse(H).data.todense())

def chain():  # its first group touches the lowest bits
    return heisenberg_chain(10, seed=2)

def middle():  # none does
    return _spins(10, [(0.4 + 0.1 * i, ((i, "x"), (i + 1, "x"))) for i in range(5, 9)] + [(0.3, ((6, "y"),))])

for model in (chain, middle):
    for form, dt, tol in FORMS:
        for run, side in ((apply, L.QOB_LEFT), (apply, L.QOB_RIGHT), (evolve, L.QOB_LEFT)):
            what = (model.__name__, form, run.__name__, side)
            err = run(model(), side, form, dt)
            assert err < tol, (what, err)
            assert status()[:2] == (0, 0), what
            bad = model()
            raise_for(lib.qob_op_prepare(ctx.ptr, handle(ctx, bad).ptr, side, form, None), ctx)
            raise_for(lib.qob_debug_shift_slot(ctx.ptr, handle(ctx, bad).ptr, side, form, N), ctx)
            err = run(bad, side, form, dt)
            rc, fl, msg = status()
            assert rc == L.QOB_ERR_ARG and fl == 2 and b"out-of-range" in msg, (what, rc, fl)
            assert err > 1e-6, what  # the skipped entries change the result
print("debug-bounds ok")
'''


def test_debug_bounds_build_checks_flips_and_row_lists():
    sys.path.insert(0, os.path.join(ROOT, "quantumopticsbase.jl_gb300"))
    import build as qob_build

    env = dict(os.environ, QOB_LIBRARY=qob_build.build(debug_bounds=True))
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "debug-bounds ok" in r.stdout

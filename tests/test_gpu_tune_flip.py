"""The tuner times the flip-form gather (times[58]) where a call of that size runs it, and only there."""
import ctypes as C

import pytest

from qobgpu import _lib as L
from qobgpu.device import get_context, handle, raise_for
from qobgpu.hamiltonians import heisenberg_chain
from test_gpu_flip import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spins,cols,side,runs", [(8, 4, L.QOB_LEFT, False), (10, 15, L.QOB_LEFT, False),
                                                   (10, 16, L.QOB_LEFT, True), (8, 4, L.QOB_RIGHT, True),
                                                   (8, 1, L.QOB_RIGHT, False)])
def test_flip_kernel_is_timed_where_it_runs(spins, cols, side, runs):
    ctx, H = get_context(0), heisenberg_chain(spins, seed=8)
    times, chosen = (C.c_double * 59)(), C.c_int()
    raise_for(L.lib().qob_op_tune_ex(ctx.ptr, handle(ctx, H).ptr, side, L.QOB_C128, cols, times, 59, C.byref(chosen)), ctx)
    assert (times[58] > 0) == runs, times[58]
    assert runs or not (chosen.value >> 29) & 1
    _check(H, cols, "left" if side == L.QOB_LEFT else "right", 0.3, 160 + spins)

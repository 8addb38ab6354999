"""A recorded call keeps the workspace it was recorded with: larger calls of the same context,
which make its buffers grow, leave the graph's own as they are."""
import ctypes as C

import numpy as np
import pytest

import qobgpu as Q
from helpers import rel_l2
from qobgpu import _lib as L
from qobgpu.device import Context, _leaf, raise_for
from test_gpu_slices import _dense, _device, _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("c128", 1e-12), ("c64", 1e-5), ("ff", 1e-12)])
@pytest.mark.parametrize("by", ["library", "torch"])
def test_replay_after_larger_calls(form, tol, by):
    import torch

    rng, lib, ctx = Q.Rng(13), L.lib(), Context(0)  # a context whose buffers have not grown yet
    code = {"c128": L.QOB_C128, "c64": L.QOB_C64, "ff": L.QOB_C128X}[form]
    s = torch.cuda.Stream()
    sp = C.c_void_p(s.cuda_stream)

    def call(h, n, k, x, y):
        raise_for(lib.qob_mul(ctx.ptr, L.QOB_LEFT, 0, h.ptr, code, 1.0, 0.0, C.c_void_p(x.data_ptr()), n, k, n, 0.0, 0.0,
                              C.c_void_p(y.data_ptr()), n, k, n, sp), ctx)

    n, k = 400, 40
    a = _matrix(rng, n, n)
    small = (_leaf(ctx, _dense(a)), n, k, _device(rng.kets_data(n, k), form), _device(np.zeros((n, k), complex), form))
    torch.cuda.synchronize()
    call(*small)
    s.synchronize()
    g = C.c_void_p()
    if by == "library":
        raise_for(lib.qob_graph_begin(ctx.ptr, sp), ctx)
        call(*small)
        raise_for(lib.qob_graph_end(ctx.ptr, sp, C.byref(g)), ctx)
    else:
        tg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(tg, stream=s):
            call(*small)
    for n2, k2 in ((700, 300), (1500, 2500)):
        b, X = _matrix(rng, n2, n2), rng.kets_data(n2, k2)
        large = (_leaf(ctx, _dense(b)), n2, k2, _device(X, form), _device(np.zeros((n2, k2), complex), form))
        torch.cuda.synchronize()
        call(*large)
        s.synchronize()
        assert rel_l2(large[4].cpu().numpy().astype(complex), b @ X) < tol
    for _ in range(2):
        X = rng.kets_data(n, k)
        small[3].copy_(torch.as_tensor(X))
        torch.cuda.synchronize()
        if by == "library":
            raise_for(lib.qob_graph_launch(ctx.ptr, g, sp), ctx)
        else:
            with torch.cuda.stream(s):
                tg.replay()
        s.synchronize()
        assert rel_l2(small[4].cpu().numpy().astype(complex), a @ X) < tol
    if by == "library":
        lib.qob_graph_free(ctx.ptr, g)

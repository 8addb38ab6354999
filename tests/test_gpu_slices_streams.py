"""Products from digit planes (k_slice.cu) on two streams of one context: their workspace is
shared, so each starts when the one before has ended.  Every result is, to the bit, what
the call returns alone."""
import ctypes as C

import pytest

import qobgpu as Q
from qobgpu import _lib as L
from qobgpu import operators as O
from qobgpu.device import get_context, handle, raise_for
from test_gpu_slices import _dense, _matrix

pytestmark = pytest.mark.gpu


def _state(rows, cols, dt, seed):
    import torch

    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return torch.randn(cols, rows, dtype=torch.complex64, device="cuda:0", generator=g).to(dt).t()


@pytest.mark.parametrize("form", ["c128", "c64"])
@pytest.mark.parametrize("other", ["dense", "modes"])
@pytest.mark.parametrize("recorded", [False, True])
def test_two_streams(form, other, recorded):
    import torch

    # many kets: the FMA kernels would use no workspace for the dense products
    rng, lib, ctx = Q.Rng(11), L.lib(), get_context(0)
    ops = [_dense(_matrix(rng, 900, 900))]
    if other == "dense":
        ops.append(_dense(_matrix(rng, 900, 900)))
        shapes = [(900, 1500), (900, 1500)]
    else:
        bs = [Q.GenericBasis(d) for d in (99, 3, 104)]
        b = Q.tensor_basis(*bs)
        ops.append(O.LazyTensor(b, b, (1, 3), (O.Operator(bs[0], bs[0], _matrix(rng, 99, 99)),
                                               O.Operator(bs[2], bs[2], _matrix(rng, 104, 104)))))
        shapes = [(900, 1500), (len(b), 40)]
    dt, code = (torch.complex64, L.QOB_C64) if form == "c64" else (torch.complex128, L.QOB_C128)
    hs = [handle(ctx, op) for op in ops]
    streams = [torch.cuda.Stream() for _ in range(2)]
    xs = [_state(r, k, dt, i) for i, (r, k) in enumerate(shapes)]
    ys = [[torch.zeros(k, r, dtype=dt, device="cuda:0").t() for _ in range(4)] for r, k in shapes]

    def call(i, y):
        r, k = shapes[i]
        raise_for(lib.qob_mul(ctx.ptr, L.QOB_LEFT, 0, hs[i].ptr, code, 1.0, 0.0, C.c_void_p(xs[i].data_ptr()), r, k, r, 0.0,
                              0.0, C.c_void_p(y.data_ptr()), r, k, r, C.c_void_p(streams[i].cuda_stream)), ctx)

    want = []
    torch.cuda.synchronize()
    for i in range(2):
        call(i, ys[i][0])
        torch.cuda.synchronize()
        want.append(ys[i][0].clone())
    graphs = []
    if recorded:
        for i in range(2):
            for y in ys[i]:
                g, sp = C.c_void_p(), C.c_void_p(streams[i].cuda_stream)
                raise_for(lib.qob_graph_begin(ctx.ptr, sp), ctx)
                call(i, y)
                raise_for(lib.qob_graph_end(ctx.ptr, sp, C.byref(g)), ctx)
                graphs.append(g)
    for _ in range(6):
        for y in ys[0] + ys[1]:
            y.zero_()
        torch.cuda.synchronize()
        for q in range(4):
            for i in range(2):
                if recorded and (q + i) % 2:
                    raise_for(lib.qob_graph_launch(ctx.ptr, graphs[4 * i + q], C.c_void_p(streams[i].cuda_stream)), ctx)
                else:
                    call(i, ys[i][q])
        torch.cuda.synchronize()
        for i in range(2):
            for y in ys[i]:
                assert torch.equal(y, want[i])
    for g in graphs:
        lib.qob_graph_free(ctx.ptr, g)

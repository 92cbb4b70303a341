"""Reductions of one context that overlap on the GPU, because the caller gave the context another stream
in between: each has its own result, and none spoils those after it, in a replayed graph either."""
import ctypes as C

import pytest
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import _lib as L
from tensorkit_b200.backend import ReducePlan

pytestmark = pytest.mark.gpu


def test_overlapping_reductions_leave_no_trace():
    ctx = tk.get_context(0)
    lib, h = ctx.lib, ctx.handle
    n = 4_000_000
    plan = ReducePlan(ctx, [(0, n, 1, 1.0)], n)
    small = ReducePlan(ctx, [(0, 5000, 1, 2.0)], n)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    want, want_small = (x * x).sum().item(), 2 * (x[:5000] ** 2).sum().item()
    res = torch.zeros(42, 2, dtype=torch.float64, device="cuda")
    rp = lambda k: C.c_void_p(res[k].data_ptr())  # noqa: E731
    xp = C.c_void_p(x.data_ptr())
    norm2 = lambda p, k: L.check(lib.tkb_reduce_async(h, p.handle, L.TKB_NORM2, L.TKB_F64, xp, None, rp(k)), h)  # noqa: E731
    torch.cuda.synchronize()
    graph = C.c_void_p()
    L.check(lib.tkb_graph_begin(h), h)
    norm2(plan, 41)
    L.check(lib.tkb_graph_end(h, C.byref(graph)), h)
    streams = [torch.cuda.Stream() for _ in range(2)]
    try:
        for k in range(40):
            L.check(lib.tkb_ctx_set_stream(h, C.c_void_p(streams[k & 1].cuda_stream)), h)
            norm2(plan, k)
            if k % 8 == 7:
                torch.cuda.synchronize()
    finally:
        torch.cuda.synchronize()
        L.check(lib.tkb_ctx_set_stream(h, C.c_void_p(ctx.stream_handle)), h)
    tol = 1e-12  # sums of 4e6 squares in another order: about 1e-14
    assert ((res[:40, 0] - want).abs() <= tol * want).all() and (res[:40, 1] == 0).all()
    out = (C.c_double * 2)()
    for p, w in ((small, want_small), (plan, want)) * 8:
        L.check(lib.tkb_reduce(h, p.handle, L.TKB_NORM2, L.TKB_F64, xp, None, out), h)
        assert abs(out[0] - w) <= tol * w
    for _ in range(3):
        res[41].zero_()
        torch.cuda.synchronize()
        L.check(lib.tkb_graph_launch(h, graph), h)
        ctx.synchronize()
        assert abs(res[41, 0].item() - want) <= tol * want
    L.check(lib.tkb_graph_destroy(graph), h)

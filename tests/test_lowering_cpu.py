"""A lowered contraction allocates what it needs before it orders the streams: memory that the caching
allocator hands out later could still be in use by work enqueued on the caller's stream since then."""
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import tensoroperations as TO


class _Lib:
    def __init__(self, log):
        self.log = log

    def __getattr__(self, name):
        def call(*args):
            self.log.append(name)
            return 0
        return call


class _Handle:
    handle = 1


def test_allocations_precede_the_stream_order(monkeypatch):
    log = []
    new = TO.new_tensor

    def alloc(W, dtype, device):
        log.append("alloc")
        return new(W, dtype, device)

    monkeypatch.setattr(TO, "new_tensor", alloc)
    monkeypatch.setattr(TO, "gemm_plan", lambda *a: _Handle())
    V = tk.Vect({tk.U1Irrep(0): 2, tk.U1Irrep(1): 3})
    W = tk.HomSpace(tk.ProductSpace([V]), tk.ProductSpace([V]))
    A, B, C = (new(W, torch.float64, "cpu") for _ in range(3))
    ctx = type("Ctx", (), dict(lib=_Lib(log), handle=0, device=0, stream_handle=7, raw_stream=lambda self, d: 0))()
    r = TO._Recipe()
    r.W, r.swap, r.adj, r.wc, r.move_c, r.plans = W, False, (False, False), W, _Handle(), {}
    r.move = ((W, _Handle(), 0), (W, _Handle(), 0))
    TO._run_recipe(ctx, r, C, A, B, 1.0, 0.0, False)
    assert log == ["alloc"] * 3 + ["tkb_ctx_after"] + ["tkb_treetransform"] * 2 + ["tkb_grouped_gemm",
                                                                                  "tkb_treetransform", "tkb_ctx_before"]

"""Reductions over many short segments (the blocks of a tensor with many sectors, the diagonals of a trace): the
values against numpy in extended precision, around the steps of the segment search (32 and 1024) and with empty,
strided and very uneven segments; and no segment may cost a round trip of the whole launch."""
import ctypes as C

import numpy as np
import pytest
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import _lib as L
from tensorkit_b200.backend import ReducePlan

pytestmark = pytest.mark.gpu


def _segments(nseg, kind):
    rng = np.random.default_rng(nseg)
    count = {"ones": np.ones(nseg, int), "short": rng.integers(0, 6, nseg),
             "uneven": np.where(np.arange(nseg) == nseg // 2, 30000, rng.integers(0, 70, nseg))}[kind]
    stride = rng.integers(1, 4, nseg)
    off, at = [], 0
    for c, s in zip(count, stride):
        off.append(at)
        at += int(max(c, 1) * s)
    return [(o, int(c), int(s), float(w)) for o, c, s, w in zip(off, count, stride, rng.integers(1, 9, nseg))], at


def _enqueue(ctx, plan, kind, x, y, res):
    code = L.TKB_C128 if x.is_complex() else L.TKB_F64
    L.check(ctx.lib.tkb_reduce_async(ctx.handle, plan.handle, kind, code, C.c_void_p(x.data_ptr()),
                                     C.c_void_p(y.data_ptr()), C.c_void_p(res.data_ptr())), ctx.handle)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["ones", "short", "uneven"])
@pytest.mark.parametrize("nseg", [1, 2, 31, 32, 33, 1023, 1024, 1025, 1056, 5000])
def test_values(nseg, kind, cplx):
    ctx = tk.get_context(0)
    segs, n = _segments(nseg, kind)
    rng = np.random.default_rng(7)
    rnd = lambda: rng.standard_normal(n) + 1j * rng.standard_normal(n) if cplx else rng.standard_normal(n)  # noqa: E731
    x, y = rnd(), rnd()
    plan = ReducePlan(ctx, segs, n)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    idx = np.concatenate([o + s * np.arange(c) for o, c, s, _ in segs])
    w = np.concatenate([np.full(c, v) for _, c, _, v in segs]).astype(np.longdouble)
    xs, ys = (a[idx].astype(np.clongdouble if cplx else np.longdouble) for a in (x, y))
    size = float(np.sum(w * np.abs(xs) * np.abs(ys))) + float(np.sum(w * np.abs(xs) ** 2)) + float(np.sum(w * np.abs(xs)))
    for k, want in ((L.TKB_NORM2, np.sum(w * np.abs(xs) ** 2)), (L.TKB_INNER, np.sum(w * np.conj(xs) * ys)),
                    (L.TKB_TRACE, np.sum(w * xs))):
        res = torch.full((2,), 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        _enqueue(ctx, plan, k, xd, yd, res)
        ctx.synchronize()
        got = complex(*res.tolist())
        assert abs(got - complex(want)) <= 1e-13 * size + 1e-300   # a few hundred roundings of 1.1e-16 at most


def test_many_segments_are_shared_out():
    """1000 segments of one element take a few times as long as one of 1000 (7 us against 4; one CTA that walked
    them took 200 to 560)."""
    ctx = tk.get_context(0)
    x = torch.ones(1000, dtype=torch.float64, device="cuda")
    res = torch.zeros(2, dtype=torch.float64, device="cuda")
    took = []
    for segs in ([(0, 1000, 1, 1.0)], [(k, 1, 1, 1.0) for k in range(1000)]):
        plan = ReducePlan(ctx, segs, 1000)
        torch.cuda.synchronize()
        best = 1e9
        with torch.cuda.stream(ctx.stream):
            for _ in range(20):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(5):
                    _enqueue(ctx, plan, L.TKB_NORM2, x, x, res)
                b.record()
                b.synchronize()
                best = min(best, a.elapsed_time(b))
        took.append(best)
        assert res[0].item() == 1000.0
    assert took[1] <= 12 * took[0]

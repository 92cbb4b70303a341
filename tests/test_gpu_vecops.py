"""add!/scale! as one pass over the data vectors (tkb_axpby) and the single-launch reductions at
their edges: vectors of 0, 1 and odd lengths, lengths around a thread block's share, data that is
8- but not 16-byte aligned, segments that begin at odd elements, empty and strided segments, a
lazy adjoint operand, α and β with and without imaginary parts, and special values. axpby does one
rounding per product and sum, so it is within 2 ulp of numpy's two; a sum of n terms is within
1e-13 of Σ|terms| for the n used here."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import O, SU2, relerr, to_device
import tensorkit_b200 as tk
from tensorkit_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _data(n, cplx, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n)
    return x + 1j * rng.standard_normal(n) if cplx else x


@pytest.mark.parametrize("n", [0, 1, 2, 3, 255, 1023, 2047, 2048, 2049, 4099, 3_000_001])
@pytest.mark.parametrize("cplx", [False, True])
def test_axpby(n, cplx):
    ctx = tk.get_context(0)
    x, y = _data(n, cplx, 1), _data(n, cplx, 2)
    a, b = (0.7 - 0.3j, -1.25 + 0.5j) if cplx else (0.7, -1.25)
    for shift in ([0] if cplx else [0, 1]):  # 1: not 16-byte aligned
        for beta in (b, 0.0):
            xd = torch.from_numpy(np.concatenate([np.zeros(shift, x.dtype), x])).cuda()[shift:]
            yd = torch.from_numpy(np.concatenate([np.zeros(shift, x.dtype), y])).cuda()[shift:]
            if beta == 0.0:
                yd.fill_(float("nan"))  # β = 0 does not read it
            torch.cuda.synchronize()
            L.check(ctx.lib.tkb_axpby(ctx.handle, L.TKB_C128 if cplx else L.TKB_F64, n, C.c_void_p(yd.data_ptr()),
                                      C.c_void_p(xd.data_ptr()), L.tkb_scalar(complex(a).real, complex(a).imag),
                                      L.tkb_scalar(complex(beta).real, complex(beta).imag)), ctx.handle)
            ctx.synchronize()
            ref = a * x + (beta * y if beta != 0.0 else 0.0)
            bound = 2 * np.finfo(float).eps * (abs(a) * np.abs(x) + abs(beta) * np.abs(y)) + 1e-300
            assert np.all(np.abs(yd.cpu().numpy() - ref) <= bound)


def test_add_scale_tensors():
    V = O.Space({SU2(0): 3, SU2(0.5): 5, SU2(1): 2})
    W = O.Hom([V, V], [V, V])
    x, y = O.randn(W, 1, True), O.randn(W, 2, True)
    xd, yd = to_device(x), to_device(y)
    tk.add_(yd, xd, 0.5 - 1j, 2.0)
    assert relerr(yd.to_host(), (0.5 - 1j) * x.data + 2.0 * y.data) <= 1e-15
    tk.scale_(yd, -0.25j)
    assert relerr(yd.to_host(), -0.25j * ((0.5 - 1j) * x.data + 2.0 * y.data)) <= 1e-15
    adj = O.permute(x, ((1, 2), (3, 4)), adjoint=True)
    z = to_device(adj)
    tk.add_(z, tk.AdjointTensorMap(xd), 1.0, 1.0)  # stored transposed: not a flat sum
    assert relerr(z.to_host(), 2.0 * adj.data) <= 1e-12
    with pytest.raises(TypeError):
        tk.add_(yd, to_device(O.randn(W, 3, False)))
    with pytest.raises(L.TKBError):
        tk.scale_(to_device(O.randn(W, 3, False)), 1j)


SEGS = [[(0, 1, 1, 2.0)], [(1, 2, 1, 1.0), (3, 0, 1, 5.0), (4, 1, 1, 3.0)],
        [(0, 4095, 1, 1.0), (4095, 4097, 1, 2.0), (8193, 3, 1, 0.5)],
        [(7, 100, 11, 2.0), (5000, 2000, 1, 1.0)],
        [(3, 1_000_003, 1, 1.5), (1_000_100, 17, 3, 2.5)]]


@pytest.mark.parametrize("segs", SEGS, ids=["one", "tiny", "blocks", "strided", "long"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
def test_reduce_segments(segs, cplx, shift):
    from tensorkit_b200.backend import ReducePlan
    ctx = tk.get_context(0)
    n = max(o + (c - 1) * s + 1 for o, c, s, _ in segs if c)
    x, y = _data(n, cplx, 3), _data(n, cplx, 4)
    xd = torch.from_numpy(np.concatenate([np.zeros(shift, x.dtype), x])).cuda()[shift:]
    yd = torch.from_numpy(y).cuda()
    torch.cuda.synchronize()
    plan = ReducePlan(ctx, segs, n)
    for kind in (L.TKB_NORM2, L.TKB_INNER, L.TKB_TRACE):
        out = np.zeros(2)
        L.check(ctx.lib.tkb_reduce(ctx.handle, plan.handle, kind, L.TKB_C128 if cplx else L.TKB_F64,
                                   C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()),
                                   out.ctypes.data_as(C.POINTER(C.c_double))), ctx.handle)
        ref, mag = 0.0, 0.0
        for o, c, s, w in segs:
            if c == 0:
                continue
            u, v = x[o:o + (c - 1) * s + 1:s], y[o:o + (c - 1) * s + 1:s]
            t = np.abs(u) ** 2 if kind == L.TKB_NORM2 else np.conj(u) * v if kind == L.TKB_INNER else u
            ref, mag = ref + w * t.sum(), mag + w * np.abs(t).sum()
        assert abs(complex(out[0], out[1]) - ref) <= 1e-13 * mag, (kind, segs)


def test_special_values():
    V = O.Space({SU2(0): 40, SU2(0.5): 30})
    x = to_device(O.randn(O.Hom([V], [V]), 5))
    x.data[7] = float("inf")
    assert tk.norm(x) == float("inf")
    tk.scale_(x, 2.0)
    assert int(torch.isinf(x.data).sum()) == 1 and not bool(torch.isnan(x.data).any())

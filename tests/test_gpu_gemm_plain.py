"""The plain grouped GEMM at the edges of its tiles and of its work decomposition, against numpy: m and
n around 32 and 64, K around a stage of 16 (and 0, 1, long), every op, odd offsets and leading
dimensions, a base that is 8- but not 16-byte aligned, launches of few small tiles, of tiles that are
cut into K pieces, and of more tiles than resident CTAs (shares that end inside a tile), with
and without split K. Any order of summation is within (k + 4)·eps·Σ|a||b| of the exact product; the
scalars add two roundings each."""
import ctypes as C

import numpy as np
import pytest
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import _lib as L
from tensorkit_b200.backend import GemmPlan

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _op(X, op):
    return X if op == L.TKB_OP_N else X.T if op == L.TKB_OP_T else X.conj().T


def _run(shapes, cplx, ops, odd, tuning=None, alpha=0.7, beta=-1.3, shift=0, seed=0, prec=L.TKB_PLAIN):
    """shapes: (m, n, k) per block; checks C = α·op(A)·op(B) + β·C."""
    rng = np.random.default_rng(seed)
    rnd = lambda n: rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)  # noqa: E731
    rows, oa, ob, oc = [], odd, odd, odd
    for i, (m, n, k) in enumerate(shapes):
        opA, opB = ops[i % len(ops)]
        lda = (m if opA == L.TKB_OP_N else k) + odd
        ldb = (k if opB == L.TKB_OP_N else n) + odd
        ldc = m + odd
        rows.append((m, n, k, oa, ob, oc, max(lda, 1), max(ldb, 1), ldc, opA, opB))
        oa += lda * (k if opA == L.TKB_OP_N else m)
        ob += ldb * (n if opB == L.TKB_OP_N else k)
        oc += ldc * n
    A, B, Cv = rnd(oa + 1), rnd(ob + 1), rnd(oc + 1)
    put = lambda x: torch.from_numpy(np.concatenate([np.zeros(shift, x.dtype), x])).cuda()[shift:]  # noqa: E731
    Ad, Bd, Cd = put(A), put(B), put(Cv)
    torch.cuda.synchronize()
    ctx = tk.get_context(0)
    plan = GemmPlan(ctx, rows, (len(A), len(B), len(Cv)), L.TKB_C128 if cplx else L.TKB_F64, prec, 0, tuning)
    sc = lambda x: L.tkb_scalar(complex(x).real, complex(x).imag)  # noqa: E731
    for _ in range(2):  # twice: the split-K counters clear themselves
        Cd.copy_(put(Cv))
        torch.cuda.synchronize()
        L.check(ctx.lib.tkb_grouped_gemm(ctx.handle, plan.handle, C.c_void_p(Cd.data_ptr()), C.c_void_p(Ad.data_ptr()),
                                         C.c_void_p(Bd.data_ptr()), sc(alpha), sc(beta)), ctx.handle)
        ctx.synchronize()
    got = Cd.cpu().numpy()
    touched = np.zeros(len(Cv), bool)
    for m, n, k, a, b, c, lda, ldb, ldc, opA, opB in rows:
        view = lambda x, o, r, q, ld: np.lib.stride_tricks.as_strided(  # noqa: E731
            x[o:], (r, q), (x.itemsize, ld * x.itemsize))
        Am = _op(view(A, a, *((m, k) if opA == L.TKB_OP_N else (k, m)), lda), opA)
        Bm = _op(view(B, b, *((k, n) if opB == L.TKB_OP_N else (n, k)), ldb), opB)
        C0, C1 = view(Cv, c, m, n, ldc), view(got, c, m, n, ldc)
        bound = EPS * ((4 * k + 8) * abs(alpha) * (np.abs(Am) @ np.abs(Bm)) + 4 * abs(beta) * np.abs(C0)) + 1e-300
        assert np.all(np.abs(C1 - (alpha * (Am @ Bm) + beta * C0)) <= bound), (m, n, k, opA, opB)
        view(touched, c, m, n, ldc)[...] = True
    assert np.array_equal(got[~touched], Cv[~touched])  # nothing outside the blocks is written


N, T, H = L.TKB_OP_N, L.TKB_OP_T, L.TKB_OP_C
OPS = [[(N, N)], [(T, N), (N, T)], [(H, H), (T, T), (N, H)]]
EDGES = [(m, n, k) for m, n in [(1, 1), (31, 33), (32, 32), (33, 64), (64, 63), (65, 129)] for k in (0, 1, 8, 15, 17, 33)]
FEW = [(64, 64, 1000), (33, 65, 517), (3, 2, 4000)]
MANY = [(1500, 1400, 37), (700, 300, 20), (130, 70, 900), (64, 640, 5), (200, 200, 0)]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ops", OPS, ids=["NN", "TN-NT", "mixed"])
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("shapes", [EDGES, FEW, MANY], ids=["edges", "few", "many"])
def test_plain_blocks(shapes, ops, odd, cplx):
    _run(shapes, cplx, ops, odd, seed=odd)


@pytest.mark.parametrize("tuning", [(1, 4), (64, 1), (3, 8)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shapes", [FEW, MANY], ids=["few", "many"])
def test_plain_tuned(shapes, cplx, tuning):
    _run(shapes, cplx, [(N, N), (T, T)], 1, tuning, beta=0.0)


THIN = [(1, 1, 512), (1, 1, 513), (1, 1, 511), (4, 4, 3000), (2, 3, 70001), (1, 4, 2048), (5, 1, 2000), (64, 48, 40)]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ops", OPS, ids=["NN", "TN-NT", "mixed"])
@pytest.mark.parametrize("shapes", [THIN, THIN[:1], THIN[:3]], ids=["mixed", "one", "dots"])
def test_thin_blocks(shapes, ops, cplx):
    _run(shapes, cplx, ops, 1)
    _run(shapes[:6], cplx, ops, 0, beta=0.0, prec=L.TKB_SPLIT_INT8)  # thin blocks run in FP64 in either precision


def test_plain_unaligned_base():
    _run(EDGES, False, [(N, N), (T, N)], 0, shift=1)

"""Contractions lowered once per structure (spaces, index tuples, scalar types) against the
step-by-step path and the oracle: equal but distinct spaces share a recipe, transposed and
conjugated operands and every placement of the result's legs get their own, α and β reach a
destination that was passed in, recipes survive the eviction of the tables and plans they refer to,
and calls from other streams and threads see each other's results in order."""
import threading

import pytest
import torch

from helpers import O, VSU2, VU1, relerr, to_device, to_hom
import tensorkit_b200 as tk
from tensorkit_b200 import indexmanipulations as IM

pytestmark = pytest.mark.gpu
TOL = 1e-12
EXPRS = ["C[a,p,q;b] := A[a,p;c]*B[c,q;b]", "C[b,a;q,p] := A[a,p;c]*B[c,q;b]", "C[q;a,b,p] := A[a,p;c]*B[c,q;b]",
         "C[a;b] := conj(A[c,p;a])*A[c,p;b]", "C[p,q;r,s] := A[a,p;c]*conj(A[a,r;d])*A[c,q;e]*conj(A[d,s;e])"]


def _space(spaces):
    V, P = spaces()[0], spaces()[2]
    return O.Hom([V, P], [V])


def _steps(fn):
    IM.LAUNCH_LOG = []  # recording launches takes the step-by-step path
    try:
        return fn()
    finally:
        IM.LAUNCH_LOG = None


@pytest.mark.parametrize("spaces", [VU1, VSU2], ids=["U1", "SU2"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("expr", EXPRS)
def test_recipes_match_steps_and_oracle(spaces, cplx, expr):
    from tensorkit_b200.tensoroperations import parse_tensor_expr
    W = _space(spaces)
    A, B = O.randn(W, 1, cplx), O.randn(W, 2, cplx)
    _, lhs, _, fac = parse_tensor_expr(expr)
    ref = O.network(fac, lhs, {"A": A, "B": B})
    for _ in range(2):  # the second time with new, equal spaces
        Ad, Bd = to_device(A), to_device(B)
        got = tk.tensor(expr, A=Ad, B=Bd)
        old = _steps(lambda: tk.tensor(expr, A=Ad, B=Bd))
        assert got.space == to_hom(ref.W)
        assert torch.equal(got.data, old.data)
        assert relerr(got.to_host(), ref.data) <= TOL
    al = 0.5 - 1.5j if cplx else -1.5
    for op, beta in (("=", 0.0), ("+=", 1.0)):
        out = tk.TensorMap(torch.full_like(got.data, 2.0), got.space)
        tk.tensor(expr.replace(":=", op), out=out, alpha=al, A=Ad, B=Bd)
        assert relerr(out.to_host(), al * ref.data + beta * 2.0) <= TOL


def test_refusals_and_eviction():
    W = _space(VSU2)
    A, B = to_device(O.randn(W, 1)), to_device(O.randn(W, 2))
    first = tk.tensor(EXPRS[1], A=A, B=B)
    with pytest.raises(tk.SpaceMismatch):
        tk.tensor(EXPRS[1].replace(":=", "="), out=tk.TensorMap.zeros(A.space, device="cuda"), A=A, B=B)
    with pytest.raises(TypeError):
        tk.tensor(EXPRS[1], A=A, B=to_device(O.randn(W, 2, True)))
    with pytest.raises(RuntimeError):
        tk.tensor(EXPRS[1], A=tk.TensorMap(A.data.cpu(), A.space), B=tk.TensorMap(B.data.cpu(), B.space))
    ctx = tk.get_context(0)
    torch.cuda.synchronize()
    for cache in (ctx.tables, ctx.plans):  # what an LRU eviction does
        for v in cache.values():
            v.free()
        cache.clear()
    assert torch.equal(tk.tensor(EXPRS[1], A=A, B=B).data, first.data)


def test_streams_and_threads():
    W = _space(VSU2)
    A, B = O.randn(W, 3), O.randn(W, 4)
    ref = tk.tensor(EXPRS[0], A=to_device(A), B=to_device(B)).to_host()
    errs = []

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                a, b = to_device(A), to_device(B)
                a.data.mul_(float(k + 1))
                c = tk.tensor(EXPRS[0], A=a, B=b)
                c.data.div_(float(k + 1))
                errs.append(relerr(c.to_host(), ref))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(errs) == 80 and max(errs) <= TOL

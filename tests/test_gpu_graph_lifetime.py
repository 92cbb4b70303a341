"""A captured network replays into the scratch and with the tables and plans it was captured with, whatever was
planned or cleared since."""
import pytest
import torch

from helpers import O, cfg2_spaces, relerr, to_device
import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu
ENV = "En[a;b] := conj(A[c,p;a])*E[c;d]*A[d,p;b]"


def _network(seed, cplx=False):
    V, Pp = cfg2_spaces(4)
    A, E = O.randn(O.Hom([V, Pp], [V]), seed, cplx), O.randn(O.Hom([V], [V]), seed + 1, cplx)
    fac = [("A", ("c", "p", "a"), True), ("E", ("c", "d"), False), ("A", ("d", "p", "b"), False)]
    return A, E, O.network(fac, (("a",), ("b",)), {"A": A, "E": E})


def test_workspace_growth_keeps_the_captured_one():
    A, E, ref = _network(3)
    plan = tk.NetworkPlan(ENV, "split", A=to_device(A), E=to_device(E))
    assert relerr(plan.replay().to_host(), ref.data) <= 1e-12
    # products that need more scratch than any context starts with (7 slices of 2·2560² values: 92 MB), more each time
    for d in (2560, 2816):
        sp = tk.ProductSpace([tk.Vect({tk.U1Irrep(0): d})])
        X = tk.TensorMap(torch.randn(d * d, dtype=torch.float64, device="cuda"), tk.HomSpace(sp, sp))
        Y = tk.TensorMap.zeros(X.space, device="cuda")
        tk.mul_(Y, X, X, prec="split")
        want = (X.data.view(d, d) @ X.data.view(d, d)).reshape(-1)
        other = torch.full((40 << 20,), 7, dtype=torch.int8, device="cuda")  # takes up freed memory
        plan.output.data.zero_()
        torch.cuda.synchronize()
        got = plan.replay()
        plan.ctx.synchronize()
        assert relerr(got.to_host(), ref.data) <= 1e-12
        assert bool((other == 7).all())
        assert ((Y.data - want).abs().max() / want.abs().max()).item() <= 1e-12
    plan.free()


@pytest.mark.parametrize("prec", ["plain", "split"])
def test_cleared_caches_keep_what_a_graph_runs_on(prec):
    from tensorkit_b200 import backend
    tk.empty_globalcaches()
    A, E, ref = _network(7)
    plan = tk.NetworkPlan(ENV, prec, A=to_device(A), E=to_device(E))
    assert relerr(plan.replay().to_host(), ref.data) <= 1e-12
    ctx = plan.ctx
    ran = list(ctx.tables.values()) + [p for k, p in ctx.plans.items() if p.pins]
    assert len(ran) == 4 and all(v.pins for v in ran)   # two permutes, two products
    tk.empty_globalcaches()
    assert not ctx.tables and not ctx.plans and all(v.handle is not None for v in ran)
    again = tk.tensor(ENV, A=plan.inputs["A"], E=plan.inputs["E"])   # new tables beside the pinned ones
    plan.output.data.zero_()
    torch.cuda.synchronize()
    got = plan.replay()
    ctx.synchronize()
    assert relerr(got.to_host(), ref.data) <= 1e-12 and relerr(again.to_host(), ref.data) <= 1e-12
    plan.free()
    assert all(v.handle is None for v in ran) and backend.USE_LOG is None

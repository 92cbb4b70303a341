"""The register recoupling kernel (tables with several trees per group) against the staged general
kernel and the oracle, at the edges of its boxes: rows of one element, rows longer than a box,
boxes with remainders on every dim, groups of 1 to 8 source trees, groups with more (which keep the
general kernel), α/β accumulation, complex data and conjugating loads. Both kernels form
Σ_j U_ij·v_j in the same order, so their results agree bit for bit; the oracle bounds the values."""
import pytest
import torch

from helpers import O, SU2, relerr, to_device, to_hom
import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _sp(*degs, dual=False):
    return O.Space({SU2(j / 2): d for j, d in enumerate(degs) if d}, dual)


def _plaquette():  # ragged boxes, up to 4 trees
    V = _sp(7, 19, 5, 1)
    return O.Hom([V, V], [V, V])


def _long_rows():  # rows beyond one box, rows of one element
    V, W = _sp(2500, 33, 1), _sp(1, 3)
    return O.Hom([V, W, W], [W])


def _many_trees():  # up to 9 trees per group: registers and general kernel
    V = _sp(0, 3, 0, 1)
    return O.Hom([V, V, V], [V, V])


def _small():
    V = _sp(1, 2, 1)
    return O.Hom([V, V], [V, _sp(2, 1, 1, dual=True)])


CASES = [(_plaquette, [((1, 3), (2, 4)), ((1, 4), (2, 3)), ((1, 3, 2), (4,)), ((2, 3), (1, 4))]),
         (_long_rows, [((1, 3), (4, 2)), ((1,), (4, 2, 3)), ((1, 2, 4), (3,))]),
         (_many_trees, [((1, 4), (2, 5, 3)), ((1, 2, 4), (3, 5)), ((3, 1, 2), (4, 5))]),
         (_small, [((1, 3), (2, 4)), ((1,), (4, 3, 2)), ((), (1, 2, 3, 4))])]


def _both(monkeypatch, fn):
    outs = []
    for kernel in ("", "plain"):
        if kernel:
            monkeypatch.setenv("TKB_TRANSFORM_KERNEL", kernel)
        else:
            monkeypatch.delenv("TKB_TRANSFORM_KERNEL", raising=False)
        outs.append(fn())
        torch.cuda.synchronize()
    return outs


@pytest.mark.parametrize("make,perms", CASES, ids=["plaquette", "long_rows", "many_trees", "small"])
@pytest.mark.parametrize("cplx", [False, True])
def test_recoupling_kernel(monkeypatch, make, perms, cplx):
    W = make()
    t = O.randn(W, 31, cplx)
    td = to_device(t)
    alpha, beta = (0.75 - 0.5j, -1.5 + 0.25j) if cplx else (0.75, -1.5)
    for p in perms:
        ref = O.permute(t, p)
        new, old = _both(monkeypatch, lambda: tk.permute(td, p, copy=True))
        assert new.space == to_hom(ref.W)
        assert torch.equal(new.data, old.data), p
        assert relerr(new.to_host(), ref.data) <= TOL, p
        c = O.randn(W.select(p), 32, cplx)
        new, old = _both(monkeypatch, lambda: tk.permute_(to_device(c), td, p, alpha, beta))
        assert torch.equal(new.data, old.data), p
        ref = O.permute(t, p, alpha=alpha, tdst=c, beta=beta)
        assert relerr(new.to_host(), ref.data) <= TOL, p
    adj = tk.AdjointTensorMap(td)
    n1, n = W.n1(), W.n1() + W.n2()
    back = n - n1 + 1  # leg 1 of t, seen from the adjoint
    q = ((back,), tuple(i for i in range(n, 0, -1) if i != back))
    ref = O.permute(t, q, adjoint=True)
    new, old = _both(monkeypatch, lambda: tk.permute(adj, q, copy=True))
    assert torch.equal(new.data, old.data)
    assert relerr(new.to_host(), ref.data) <= TOL

"""Row copies by warps and by CTAs: the same call through the plain kernel forms α·(u·v) + β·d per
element in the same order, so the results agree bit for bit; the oracle bounds the values (1e-12).
Tables: task counts that leave the last CTA part empty, rows of odd and even length (element pairs
or single elements), tasks below and above the warp limits with few and with many tasks, rows
longer than a task, a data vector that is not 16-byte aligned."""
import pytest
import torch

from helpers import O, U1, relerr, to_device
import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _legs(deg, q):
    return O.Space({U1(i): deg for i in range(-q, q + 1)})


def _four(deg, q):
    V = _legs(deg, q)
    return O.Hom([V, V], [V, V])


def _long():
    V, P = O.Space({U1(0): 9001, U1(1): 4096, U1(2): 3}), O.Space({U1(0): 1, U1(1): 2})
    return O.Hom([V, P], [P])


CASES = {"tiny": _four(1, 2), "small_odd": _four(3, 2), "small_pairs": _four(4, 2), "medium_few": _four(20, 1),
         "medium_many": _four(17, 2), "long": _long()}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("cplx", [False, True])
def test_row_tasks(monkeypatch, name, cplx):
    W = CASES[name]
    p = ((1, 3), (2, 4)) if W.n1() + W.n2() == 4 else ((1, 3), (2,))
    t, c = O.randn(W, 41, cplx), O.randn(W.select(p), 42, cplx)
    td = to_device(t)
    alpha, beta = (0.75 - 0.5j, -1.5 + 0.25j) if cplx else (0.75, -1.5)

    def run():
        outs = [tk.permute(td, p, copy=True).data, tk.permute_(to_device(c), td, p, alpha, beta).data]
        if not cplx:  # one element off the 16-byte boundary
            buf = torch.empty(td.data.numel() + 1, dtype=td.data.dtype, device=td.data.device)
            buf[1:] = td.data
            outs.append(tk.permute(tk.TensorMap(buf[1:], td.space), p, copy=True).data)
        torch.cuda.synchronize()
        return outs

    monkeypatch.delenv("TKB_TRANSFORM_KERNEL", raising=False)
    new = run()
    monkeypatch.setenv("TKB_TRANSFORM_KERNEL", "plain")
    for a, b in zip(new, run()):
        assert torch.equal(a, b)
    assert relerr(new[0].cpu().numpy(), O.permute(t, p).data) <= TOL
    assert relerr(new[1].cpu().numpy(), O.permute(t, p, alpha=alpha, tdst=c, beta=beta).data) <= TOL

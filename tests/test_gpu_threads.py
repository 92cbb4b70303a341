"""Host threads that share a context: split products (slicing and products go through the context's
workspace) and reductions, enqueued between each other, each with its own operands on its own stream."""
import threading

import pytest
import torch

from helpers import O, cfg2_spaces, relerr, to_device, to_hom
import tensorkit_b200 as tk
from tensorkit_b200.linalg import gemm_plan

pytestmark = pytest.mark.gpu


def test_split_products_and_norms_from_threads():
    V, Pp = cfg2_spaces(4)
    cases = []
    for k in range(4):
        cplx = k % 2 == 1
        A, B = O.randn(O.Hom([V, Pp], [V]), 2 * k + 1, cplx), O.randn(O.Hom([V], [V]), 2 * k + 2, cplx)
        ref = O.mul(A, B)
        Ad, Bd = to_device(A), to_device(B)
        C = tk.TensorMap.zeros(to_hom(ref.W), dtype=Ad.dtype, device="cuda")
        plan = gemm_plan(tk.get_context(0), C, Ad, Bd, "split")
        tk.mul_(C, Ad, Bd, 1.0, 0.0, prec="split")
        assert plan.flops >= 8e6 and 7 in plan.last_slices()[0]
        cases.append((Ad, Bd, ref, tk.norm(Ad)))
    torch.cuda.synchronize()
    errs, nerrs, fails = [], [], []

    def work(k):
        try:
            Ad, Bd, ref, want = cases[k]
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(30):
                    C = tk.TensorMap.zeros(to_hom(ref.W), dtype=Ad.dtype, device="cuda")
                    tk.mul_(C, Ad, Bd, 1.0, 0.0, prec="split")
                    nerrs.append(abs(tk.norm(Ad) - want) / want)
                    errs.append(relerr(C.to_host(), ref.data))
        except Exception as e:  # noqa: BLE001
            fails.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fails
    # the products to the split tolerance; the same reduction twice gives the same bits
    assert len(errs) == 120 and max(errs) <= 1e-12 and max(nerrs) == 0.0

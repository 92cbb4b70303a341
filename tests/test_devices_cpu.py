"""Operands that one launch cannot read together are refused on the host, before anything is enqueued: on different
GPUs (a launch takes its context from one operand, so another GPU's pointer would be an invalid access) or of
different scalar types (the other vector would be read as the first one's type, past its end)."""
import pytest
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import indexmanipulations as IM
from tensorkit_b200 import linalg as LA
from tensorkit_b200 import tensoroperations as TO


class _Data:
    """Stands in for a data vector on GPU `index`."""
    is_cuda = True
    dtype = torch.float64

    def __init__(self, n, index):
        self.n, self.device = n, torch.device("cuda", index)

    def get_device(self):
        return self.device.index

    def dim(self):
        return 1

    def numel(self):
        return self.n

    def is_complex(self):
        return False


@pytest.fixture
def on(monkeypatch):
    def no_context(device=None):
        raise AssertionError("a context was asked for")

    for mod in (IM, LA, TO):
        monkeypatch.setattr(mod, "get_context", no_context)
    V = tk.Vect({tk.U1Irrep(0): 2, tk.U1Irrep(1): 3})
    W = tk.HomSpace(tk.ProductSpace([V]), tk.ProductSpace([V]))
    return lambda index: tk.TensorMap(_Data(W.dim(), index), W)


P = ((1,), (2,))
CALLS = {
    "mul": lambda a, b: tk.mul_(a, a, b),
    "inner": lambda a, b: tk.inner(a, b),
    "add": lambda a, b: tk.add_(a, b),
    "add_adjoint": lambda a, b: IM.add_transform_(a, tk.AdjointTensorMap(b), P, None),
    "contract": lambda a, b: TO.tensorcontract(a, P, False, b, P, False, P),
    "contract_adjoint": lambda a, b: TO.tensorcontract(a, P, False, b, ((2,), (1,)), True, P),
    "contract_into": lambda a, b: TO.tensorcontract_(b, a, P, False, a, P, False, P),
    "expression": lambda a, b: tk.tensor("C[x;z] := A[x;y]*B[y;z]", A=a, B=b),
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_operands_on_two_gpus_are_refused(on, monkeypatch, call):
    if call == "contract_into":  # the recipe belongs to the operands' GPU; the destination is elsewhere
        r = type("Recipe", (), {"W": on(0).space})()
        monkeypatch.setattr(TO, "_recipe", lambda *a: (None, r))
    with pytest.raises(RuntimeError, match="different devices"):
        CALLS[call](on(0), on(1))


@pytest.mark.parametrize("first", [torch.float64, torch.complex128])
def test_inner_of_two_scalar_types_is_refused(on, first):
    x, y = on(0), on(0)
    x.data.dtype = first
    y.data.dtype = torch.complex128 if first == torch.float64 else torch.float64
    with pytest.raises(TypeError, match="scalar type"):
        tk.inner(x, y)

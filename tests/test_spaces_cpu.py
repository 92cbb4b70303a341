"""Spaces across processes: hashes of text differ from one to the next, loaded spaces must not."""
import gc
import os
import pickle
import subprocess
import sys

import tensorkit_b200 as tk
from tensorkit_b200 import spaces
from tensorkit_b200.spaces import GradedSpace, HomSpace, ProductSpace

WRITE = """
import pickle, sys
sys.path.insert(0, sys.argv[1])
import tensorkit_b200 as tk
V = tk.Vect({tk.U1Irrep(0): 3, tk.U1Irrep(-1): 2}, True)
S = tk.Vect({tk.ProductSector(tk.U1Irrep(1), tk.SU2Irrep(twice=1)): 4})
W = tk.HomSpace(tk.ProductSpace([V]), tk.ProductSpace([V]))
W.adjoint(), W.dim(), V.dual(), W.select(((1,), (2,)))
sys.stdout.buffer.write(pickle.dumps((V, S, W)))
"""


def _spaces():
    V = tk.Vect({tk.U1Irrep(0): 3, tk.U1Irrep(-1): 2}, True)
    S = tk.Vect({tk.ProductSector(tk.U1Irrep(1), tk.SU2Irrep(twice=1)): 4})
    return V, S, tk.HomSpace(tk.ProductSpace([V]), tk.ProductSpace([V]))


def test_pickled_in_another_process():
    pkg = os.path.dirname(os.path.dirname(os.path.abspath(tk.__file__)))
    for seed in ("1", "2"):
        raw = subprocess.run([sys.executable, "-c", WRITE, pkg], env=dict(os.environ, PYTHONHASHSEED=seed),
                             check=True, capture_output=True).stdout
        for got, want in zip(pickle.loads(raw), _spaces()):
            assert got == want and hash(got) == hash(want) and repr(got) == repr(want)
            assert got.dual() == want.dual()


def test_fields_of_an_earlier_pickle():
    """State that holds the fields alone, with another process's hashes and without the kept results."""
    V, _, W = _spaces()

    def bare(o, names):
        n = type(o).__new__(type(o))
        n.__setstate__((None, dict({k: getattr(o, k) for k in names}, _h=1)))
        return n

    v = bare(V, ("_keys", "_degs", "dual_flag", "_unit", "_sectors", "_dimmap"))
    w = bare(W, ("codomain", "domain"))
    assert isinstance(v, GradedSpace) and isinstance(w, HomSpace) and isinstance(w.codomain, ProductSpace)
    assert v == V and v.dual() == V.dual() and w == W and w.dim() == W.dim() and w.adjoint() == W.adjoint()
    s = bare(tk.SU2Irrep(twice=3), ("j2",))
    assert s == tk.SU2Irrep(twice=3) and hash(s) == hash(tk.SU2Irrep(twice=3))


def test_permuting_to_and_fro_keeps_no_chain():
    """A loop x = permute(x, p) comes back to the same spaces instead of making two more every time."""
    V, P = tk.Vect({tk.U1Irrep(0): 3, tk.U1Irrep(1): 2}), tk.Vect({tk.U1Irrep(0): 1, tk.U1Irrep(1): 1})
    W = tk.HomSpace(tk.ProductSpace([V, P]), tk.ProductSpace([V, P]))
    live = lambda: sum(type(o) is HomSpace for o in gc.get_objects())  # noqa: E731
    x, keep = W, W  # the first space stays alive, as the caches' keys hold it
    x = x.permute(((1, 3), (2, 4))).permute(((1, 3), (2, 4)))
    gc.collect()
    before = live()
    for _ in range(500):
        x = x.permute(((1, 3), (2, 4)))
        x = x.permute(((1, 3), (2, 4)))
    gc.collect()
    assert x == keep and live() - before <= 4


def test_selections_are_bounded():
    P = tk.Vect({tk.U1Irrep(0): 1})
    for d in range(1, spaces._MAX_SELECTED + 20):
        V = tk.Vect({tk.U1Irrep(0): d})
        W = tk.HomSpace(tk.ProductSpace([V, P]), tk.ProductSpace([V]))
        S = W.permute(((2, 1), (3,)))
        assert S is W.permute(((2, 1), (3,))) and S.codomain.spaces == (P, V)
        assert len(spaces._SELECTED) <= spaces._MAX_SELECTED

"""Caches of tables, plans and lowered contractions: what a lowered contraction keeps using is not the first to be
freed, although it holds its entries and looks none of them up."""
import torch

import tensorkit_b200 as tk
from tensorkit_b200 import tensoroperations as TO
from tensorkit_b200.backend import _LRU


class _Entry:
    handle = 1

    def free(self):
        self.handle = None


class _Lib:
    def __getattr__(self, name):
        return lambda *args: 0


def _cache(n):
    return _LRU(n, lambda e: e.free())


def test_least_recently_used_goes_first():
    c = _cache(3)
    a, b, d = (c.get_or(k, _Entry) for k in "abd")
    c.get_or("a", _Entry)
    c.get_or("e", _Entry)
    assert list(c) == ["d", "a", "e"] and b.handle is None and a.handle == d.handle == 1


def test_marked_entries_go_to_the_back_once():
    c = _cache(3)
    a, b, d = (c.get_or(k, _Entry) for k in "abd")
    a.used = b.used = d.used = True
    e = c.get_or("e", _Entry)   # every other entry is marked: the oldest goes, not the new one
    assert sorted(c) == ["b", "d", "e"] and a.handle is None and e.handle == 1
    c.get_or("f", _Entry)
    assert "f" in c and len(c) == 3


def test_entries_of_a_lowered_contraction_stay(monkeypatch):
    tables, plans, recipes = _cache(8), _cache(4), _LRU(4)
    monkeypatch.setattr(TO, "gemm_plan", lambda *a: plans.get_or("hot", _Entry))
    V = tk.Vect({tk.U1Irrep(0): 2, tk.U1Irrep(1): 3})
    W = tk.HomSpace(tk.ProductSpace([V]), tk.ProductSpace([V]))
    new = lambda: TO.new_tensor(W, torch.float64, "cpu")  # noqa: E731
    A, B, C = new(), new(), new()
    ctx = type("Ctx", (), dict(lib=_Lib(), handle=0, device=0, stream_handle=7, raw_stream=lambda self, d: 0,
                               tables=tables, plans=plans, recipes=recipes))()
    made = []

    def make(*args):
        made.append(args)
        r = TO._Recipe()
        r.W, r.swap, r.adj, r.wc, r.plans = W, False, (False, False), W, {}
        t = [tables.get_or(("hot", k), _Entry) for k in range(3)]
        r.move, r.move_c = ((W, t[0], 0), (W, t[1], 0)), t[2]
        return r

    class Cuda:  # what `_recipe` asks of a data vector
        is_cuda, dtype, device = True, torch.float64, torch.device("cuda", 0)

        def get_device(self):
            return 0

    monkeypatch.setattr(TO, "_make_recipe", make)
    monkeypatch.setattr(TO, "get_context", lambda i: ctx)
    X = type("X", (), dict(data=Cuda(), space=W))()
    p = ((1,), (2,))
    for k in range(40):
        _, r = TO._recipe(X, p, False, X, p, False, p)
        TO._run_recipe(ctx, r, C, A, B, 1.0, 0.0, False)
        tables.get_or(("cold", k), _Entry)
        plans.get_or(("cold", k), _Entry)
        recipes.get_or(("cold", k), _Entry)
    assert len(made) == 1 and r.usable() and plans["hot"].handle == 1
    assert len(tables) == 8 and len(plans) == 4 and len(recipes) == 4


def test_pinned_entries_outlive_their_cache():
    """What a captured graph runs on is freed when the graph goes, not when it leaves the cache."""
    from tensorkit_b200.backend import Owned

    class Table(Owned):
        handle = 1

        def free(self):
            self.handle = None

    c = _LRU(1, lambda e: e.drop())
    a = c.get_or("a", Table)
    a.pin()
    a.pin()     # two graphs, or twice in one
    b = c.get_or("b", Table)
    c.get_or("d", Table)
    assert a.handle == 1 and b.handle is None and list(c) == ["d"]
    a.unpin()
    assert a.handle == 1
    a.unpin()
    assert a.handle is None
    e = c.get_or("e", Table)
    e.pin()
    e.unpin()
    assert e.handle == 1  # still in its cache

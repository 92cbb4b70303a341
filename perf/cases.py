"""The work that a user of this package has it do, as cases that a timing program can run.

Every case goes through the package's public entry points: `@tensor` expressions evaluated at once
(`tk.tensor`) or captured once and replayed (`tk.NetworkPlan`), `permute`, the vector-space
operations of a Krylov solver, partial traces, and the pullback of a network. Spaces are those of
the contraction workloads of the tests and the benchmark, with their degeneracies scaled; a scale
that is not a whole number gives odd and ragged block sizes.

Kinds of cases (`kind`):
  pair      U(1): C[a,p,q;b] := A[a,p;c]*B[c,q;b] and its regrouping permute(C, ((1,3),(2,4)))
  env       SU(2) environment update En[a;b] := conj(A[c,p;a])*E[c;d]*A[d,p;b]
  heff      U(1) two-site effective Hamiltonian applied to a two-site tensor
  grad      U(1) x SU(2): forward and pullback of f[] := EL[a;c]*A[c,p;d]*ER[d;b]*conj(A[a,p;b])
  recouple  SU(2): permute(T, ((1,3),(2,4))) of a four-leg tensor (several trees per block)
  regroup   U(1): permute of a two-site tensor or of its lazy adjoint
  krylov    SU(2): one Gram-Schmidt step of a Lanczos iteration on a two-site tensor
  ptrace    SU(2): rho[a;b] := X[a,s;b,s]

`exact` evaluates the same formulas with plain torch in 64 bits on its own reading of the storage
layout (blocks of the coupled sectors in sector order, column-major, rows and columns ordered by
fusion trees whose last leg varies slowest).
"""
import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "tensorkit.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tensorkit_b200 as tk  # noqa: E402

DEV = "cuda:0"

ENV = "En[a;b] := conj(A[c,p;a])*E[c;d]*A[d,p;b]"
HEFF = "y[a,p,q;b] := L[a,w;c]*x[c,r,s;d]*W1[w,p;r,v]*W2[v,q;s,u]*R[d,u;b]"
PAIR = "C[a,p,q;b] := A[a,p;c]*B[c,q;b]"
GRAD = "f[] := EL[a;c]*A[c,p;d]*ER[d;b]*conj(A[a,p;b])"
TRACE = "rho[a;b] := X[a,s;b,s]"


def listed():
    return [
        # the smallest calls: a contraction and a regrouping of a few thousand elements, evaluated
        # at once (what a test, a small DMRG or a first sweep does thousands of times)
        dict(name="pair_u1_small", kind="pair", deg=8, qmax=3, dtype="f64"),
        # an ordinary environment update evaluated at once, at a small bond dimension
        dict(name="env_su2_small", kind="env", mult=1.0, dtype="f64", precision="plain", mode="eager"),
        # the same contraction at a production bond dimension, captured and replayed as a sweep does,
        # in both precisions that a caller can choose
        dict(name="env_su2_large", kind="env", mult=8.0, dtype="f64", precision="plain", mode="graph"),
        dict(name="env_su2_large_split", kind="env", mult=8.0, dtype="f64", precision="split", mode="graph"),
        # time evolution works on complex tensors; ragged odd blocks
        dict(name="env_su2_c128", kind="env", mult=5.3, dtype="c128", precision="plain", mode="eager"),
        # the matrix-vector product of a two-site DMRG eigensolver: many uneven blocks, large permutes
        # and tall-skinny products with the MPO tensors
        dict(name="heff_u1", kind="heff", deg=256, qmax=10, precision="plain"),
        dict(name="heff_u1_split", kind="heff", deg=256, qmax=10, precision="split"),
        # differentiation: forward and backward of a scalar loss, complex, product sectors
        dict(name="grad_u1su2_c128", kind="grad", deg=64),
        # regrouping a plaquette tensor between the steps of a tensor renormalisation
        dict(name="recouple_su2", kind="recouple", mult=2.7, jmax=4, dtype="f64"),
        # conjugate of a two-site tensor brought into matrix form (transposing, complex)
        dict(name="regroup_u1_adjoint", kind="regroup", deg=1201, qmax=8, dtype="c128", adjoint=True),
        # vector arithmetic of an eigensolver between two matrix-vector products
        dict(name="krylov_su2", kind="krylov", mult=25.3, dtype="f64"),
        # reduced density matrix of a large bipartite operator
        dict(name="ptrace_su2", kind="ptrace", mult=1.9, wmult=2.0, dtype="f64"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pair", "env", "env", "heff", "heff", "grad", "recouple", "regroup", "krylov", "ptrace"])
    dtype = rng.choice(["f64", "c128"])
    r2 = lambda x: round(x, 2)  # noqa: E731
    if kind == "pair":
        return dict(kind=kind, deg=int(round(_log(rng, 3, 60))), qmax=rng.randint(2, 5), dtype=dtype)
    if kind == "env":
        return dict(kind=kind, mult=r2(_log(rng, 0.5, 8.0)), dtype=dtype, precision=rng.choice(["plain", "split"]),
                    mode=rng.choice(["eager", "graph"]))
    if kind == "heff":
        return dict(kind=kind, deg=int(round(_log(rng, 12, 256))), qmax=rng.randint(4, 10),
                    precision=rng.choice(["plain", "split"]))
    if kind == "grad":
        return dict(kind=kind, deg=int(round(_log(rng, 6, 64))))
    if kind == "recouple":
        return dict(kind=kind, mult=r2(_log(rng, 0.4, 2.0)), jmax=rng.randint(2, 4), dtype=dtype)
    if kind == "regroup":
        return dict(kind=kind, deg=int(round(_log(rng, 30, 1000))), qmax=rng.randint(3, 8), dtype=dtype,
                    adjoint=rng.random() < 0.5)
    if kind == "krylov":
        return dict(kind=kind, mult=r2(_log(rng, 0.5, 18.0)), dtype=dtype)
    return dict(kind=kind, mult=r2(_log(rng, 0.3, 1.8)), wmult=r2(_log(rng, 0.5, 2.0)), dtype=dtype)


# ---- spaces ------------------------------------------------------------------------------------
# A sector is a tuple: (q,) of U(1), (2j,) of SU(2), (q, 2j) of their product; `sym` names which. A
# leg is (degeneracies {sector: n}, dual flag).
def _scaled(degs, mult):
    return {s: max(1, int(round(d * mult))) for s, d in degs.items()}


def _gauss(deg, qmax, width=18.0):
    return {(q,): max(1, int(round(deg * math.exp(-q * q / width)))) for q in range(-qmax, qmax + 1)}


_SPIN_V = {(j,): d for j, d in enumerate([32, 48, 40, 24, 12, 6, 2])}
_SPIN_W = {(0,): 6, (1,): 5, (2,): 3}
_PLAQ = {(0,): 7, (1,): 11, (2,): 8, (3,): 5, (4,): 3}


def _shapes(case):
    """(sym, {name: (codomain legs, domain legs)}) of the case's inputs."""
    k = case["kind"]
    leg = lambda d, dual=False: (d, dual)  # noqa: E731
    if k == "pair":
        V = {(q,): case["deg"] for q in range(-case["qmax"], case["qmax"] + 1)}
        P = {(q,): 1 for q in (-1, 0, 1)}
        W = ((leg(V), leg(P)), (leg(V),))
        return "U1", {"A": W, "B": W}
    if k == "env":
        V, P = _scaled(_SPIN_V, case["mult"]), {(1,): 1}
        return "SU2", {"A": ((leg(V), leg(P)), (leg(V),)), "E": ((leg(V),), (leg(V),))}
    if k == "heff":
        V, P, W = _gauss(case["deg"], case["qmax"]), {(0,): 1, (1,): 1}, {(-1,): 2, (0,): 3, (1,): 2}
        return "U1", {"L": ((leg(V), leg(W, True)), (leg(V),)), "x": ((leg(V), leg(P), leg(P)), (leg(V),)),
                      "W1": ((leg(W), leg(P)), (leg(P), leg(W))), "W2": ((leg(W), leg(P)), (leg(P), leg(W))),
                      "R": ((leg(V), leg(W)), (leg(V),))}
    if k == "grad":
        V = {(q, j): max(1, int(round(case["deg"] * math.exp(-(q * q + j) / 4)))) for q in range(-2, 3) for j in range(4)}
        P = {(1, 1): 1, (-1, 1): 1}
        return "U1xSU2", {"A": ((leg(V), leg(P)), (leg(V),)), "EL": ((leg(V),), (leg(V),)), "ER": ((leg(V),), (leg(V),))}
    if k == "recouple":
        V = _scaled({s: d for s, d in _PLAQ.items() if s[0] <= case["jmax"]}, case["mult"])
        return "SU2", {"T": ((leg(V), leg(V)), (leg(V), leg(V)))}
    if k == "regroup":
        V, P = _gauss(case["deg"], case["qmax"]), {(-1,): 1, (0,): 1, (1,): 1}
        return "U1", {"x": ((leg(V), leg(P), leg(P)), (leg(V),))}
    if k == "krylov":
        V, P = _scaled(_SPIN_V, case["mult"]), {(1,): 1}
        W = ((leg(V), leg(P), leg(P)), (leg(V),))
        return "SU2", {"v": W, "w": W}
    V, W = _scaled(_SPIN_V, case["mult"]), _scaled(_SPIN_W, case["wmult"])
    return "SU2", {"X": ((leg(V), leg(W)), (leg(V), leg(W)))}


def _dtype(case):
    return torch.complex128 if case.get("dtype") == "c128" or case["kind"] == "grad" else torch.float64


def _tk_sector(sym, s):
    if sym == "U1":
        return tk.U1Irrep(s[0])
    if sym == "SU2":
        return tk.SU2Irrep(twice=s[0])
    return tk.ProductSector(tk.U1Irrep(s[0]), tk.SU2Irrep(twice=s[1]))


def _tk_hom(sym, W):
    sp = lambda leg: tk.Vect({_tk_sector(sym, s): d for s, d in leg[0].items()}, leg[1])  # noqa: E731
    return tk.HomSpace(tk.ProductSpace([sp(x) for x in W[0]]), tk.ProductSpace([sp(x) for x in W[1]]))


# ---- the storage layout, read independently (sizes, work counts and exact values) ---------------
def _key(sym, s):
    u = lambda q: (abs(q), q < 0)  # noqa: E731
    return u(s[0]) if sym == "U1" else (s[0],) if sym == "SU2" else (u(s[0]), s[1])


def _dual(sym, s):
    return (-s[0],) if sym == "U1" else s if sym == "SU2" else (-s[0], s[1])


def _dim(sym, s):
    return 1 if sym == "U1" else s[-1] + 1


def _fuse(sym, a, b):
    if sym == "U1":
        return [(a[0] + b[0],)]
    spins = range(abs(a[-1] - b[-1]), a[-1] + b[-1] + 1, 2)
    return [(j,) for j in spins] if sym == "SU2" else [(a[0] + b[0], j) for j in spins]


def _leg_sectors(sym, leg):
    """(sector on the leg, degeneracy) in the order of the stored keys."""
    keys = sorted(leg[0], key=lambda s: _key(sym, s))
    return [(_dual(sym, s) if leg[1] else s, leg[0][s]) for s in keys]


def _trees(sym, legs):
    """{coupled sector: [(sectors, degeneracies)]} over the fusion trees of the legs, in order (the
    last leg slowest, then the inner line)."""
    first = {}
    for s, d in _leg_sectors(sym, legs[0]):
        first[s] = [((s,), (d,))]
    cur = first
    for leg in legs[1:]:
        nxt = {}
        for s, d in _leg_sectors(sym, leg):
            # the inner lines of c come in the order of the fusion products of c and dual(s)
            reach = sorted({c for a in cur for c in _fuse(sym, a, s)}, key=lambda c: _key(sym, c))
            for c in reach:
                for a in _fuse(sym, c, _dual(sym, s)):
                    for secs, degs in cur.get(a, ()):
                        nxt.setdefault(c, []).append((secs + (s,), degs + (d,)))
        cur = nxt
    return cur


def _prod(xs):
    r = 1
    for x in xs:
        r *= x
    return r


@lru_cache(maxsize=64)
def _layout_cached(sym, W):
    cod, dom = [[(dict(d), f) for d, f in side] for side in W]
    rows, cols = _trees(sym, cod), _trees(sym, dom)
    out, off = {}, 0
    for c in sorted(set(rows) & set(cols), key=lambda s: _key(sym, s)):
        r, n1 = [], 0
        for secs, degs in rows[c]:
            r.append((secs, degs, n1))
            n1 += _prod(degs)
        q, n2 = [], 0
        for secs, degs in cols[c]:
            q.append((secs, degs, n2))
            n2 += _prod(degs)
        out[c] = (off, n1, n2, r, q)
        off += n1 * n2
    return out, off


def _layout(sym, W):
    """({coupled: (offset, rows, columns, row trees, column trees)}, length); a tree is (sectors,
    degeneracies, first row or column)."""
    return _layout_cached(sym, tuple(tuple((tuple(sorted(d.items())), f) for d, f in side) for side in W))


def _block(x, b):
    return x[b[0]:b[0] + b[1] * b[2]].view(b[2], b[1]).T


def _sub(x, b, row, col):
    """Strided view of one sub-block: dims of the codomain legs, then of the domain legs."""
    size = row[1] + col[1]
    strides, s = [], 1
    for d in row[1]:
        strides.append(s)
        s *= d
    s = b[1]
    for d in col[1]:
        strides.append(s)
        s *= d
    return x.as_strided(size, strides, x.storage_offset() + b[0] + row[2] + col[2] * b[1])


# ---- inputs and passes ----------------------------------------------------------------------------
def _random(n, dtype, gen):
    return torch.randn(n, dtype=dtype, device=DEV, generator=gen)


def _inputs(case, seed):
    """{name: flat data vector}: independent normals from the seed, in the order of the names."""
    sym, shapes = _shapes(case)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return {n: _random(_layout(sym, W)[1], _dtype(case), gen) for n, W in shapes.items()}


def prepare(case, seed):
    sym, shapes = _shapes(case)
    data = _inputs(case, seed)
    t = {n: tk.TensorMap(data[n], _tk_hom(sym, shapes[n])) for n in shapes}
    state = {"case": case, "t": t}
    k = case["kind"]
    if k == "heff" or case.get("mode") == "graph":
        expr = HEFF if k == "heff" else ENV
        state["plan"] = tk.NetworkPlan(expr, precision=case["precision"], **t).capture()
    if k == "grad":
        state["one"] = torch.ones(1, dtype=_dtype(case), device=DEV)
    if k == "krylov":
        state["z"] = t["w"].similar()
    if k in ("recouple", "regroup"):  # large tensors are permuted into storage that is kept
        src, p = _permutation(case, t)
        state["out"] = tk.TensorMap.empty(src.space.permute(p), _dtype(case), DEV)
    return state


def _permutation(case, t):
    if case["kind"] == "recouple":
        return t["T"], ((1, 3), (2, 4))
    if case["adjoint"]:  # x' has legs (b; a, p, q): back to (a, p; q, b)
        return t["x"].adjoint(), ((2, 3), (4, 1))
    return t["x"], ((1, 2), (4, 3))


def run(state):
    case, t = state["case"], state["t"]
    k = case["kind"]
    if "plan" in state:
        return state["plan"].replay().data
    if k == "pair":
        C = tk.tensor(PAIR, **t)
        return [C.data, tk.permute(C, ((1, 3), (2, 4))).data]
    if k == "env":
        with tk.using_precision(case["precision"]):
            return tk.tensor(ENV, **t).data
    if k == "grad":
        from tensorkit_b200.chainrules import network_with_pullback
        f, pullback = network_with_pullback(GRAD, **t)
        g = pullback(tk.TensorMap(state["one"], f.space))
        return [f.data, g["A"].data, g["EL"].data, g["ER"].data]
    if k in ("recouple", "regroup"):
        src, p = _permutation(case, t)
        return tk.permute_(state["out"], src, p).data
    if k == "krylov":
        v, w, z = t["v"], t["w"], state["z"]
        a = tk.inner(v, w)
        tk.add_(z, w, 1.0, 0.0)
        tk.add_(z, v, -a, 1.0)
        n = tk.norm(z)
        tk.scale_(z, 1.0 / n)
        return [float(a.real), float(a.imag), n, z.data]
    return tk.tensor(TRACE, **t).data


# ---- work of one pass -----------------------------------------------------------------------------
def _heff_flops(V, P, W):
    """Multiply-adds of the four pairwise products, each counted over the allowed charges."""
    g = lambda d, q: d.get((q,), 0)  # noqa: E731
    qs = lambda d: [s[0] for s in d]  # noqa: E731
    n = 0
    for a in qs(V):
        for w in qs(W):
            c = a - w  # L: a - w = c
            for r in qs(P):
                for s in qs(P):
                    m = g(V, a) * g(W, w) * g(V, c + r + s)
                    n += m * g(V, c)  # L x
                    if g(V, c):
                        n += m * sum(g(W, w + p - r) for p in qs(P))  # W1
        for p in qs(P):
            for v in qs(W):
                for s in qs(P):
                    m = g(V, a) * g(W, v) * g(V, a + p - v + s)
                    n += m * sum(g(W, v + q - s) for q in qs(P))  # W2
            for q in qs(P):
                n += g(V, a) * g(V, a + p + q) * sum(g(W, u) * g(V, a + p + q - u) for u in qs(W))  # R
    return 2.0 * n


def work(case):
    sym, shapes = _shapes(case)
    el = 16 if _dtype(case) == torch.complex128 else 8
    mul = 8.0 if el == 16 else 2.0  # flops of one multiply-add
    size = {n: _layout(sym, W)[1] for n, W in shapes.items()}
    k = case["kind"]
    if k == "pair":
        lay, _ = _layout(sym, shapes["A"])
        V, P = shapes["A"][0][0], shapes["A"][0][1]
        out = _layout(sym, ((V, P, P), (V,)))[1]
        n = 0
        for c, b in lay.items():  # A[a,p;c] B[c,q;b]: the rows of block c meet c and every (q, b)
            n += b[1] * b[2] * sum(d * V[0].get((c[0] + q,), 0) for (q,), d in P[0].items())
        return {"bytes": el * (size["A"] + size["B"] + 3 * out), "flops": mul * n}
    if k == "env":
        V = shapes["A"][0][0][0]
        rows = lambda c: sum(V.get((c + s,), 0) for s in (-1, 1))  # noqa: E731
        n = sum(2 * d * d * rows(c) for (c,), d in V.items())
        return {"bytes": el * (size["A"] + 2 * size["E"]), "flops": mul * n}
    if k == "heff":
        V, P, W = shapes["x"][0][0][0], shapes["x"][0][1][0], shapes["W1"][0][0][0]
        return {"bytes": el * (sum(size.values()) + size["x"]), "flops": _heff_flops(V, P, W)}
    if k == "grad":
        lay, _ = _layout(sym, shapes["A"])
        V = shapes["A"][0][0][0]
        n = 0
        for c, (_, n1, n2, rows, _) in lay.items():
            n += sum(V[r[0][0]] * r[1][0] for r in rows) * n2 + n1 * n2 * n2 + n1 * n2
        # each product costs as much again for either operand's gradient
        return {"bytes": 2 * el * sum(size.values()), "flops": 3 * mul * n}
    if k in ("recouple", "regroup"):
        n = size["T"] if k == "recouple" else size["x"]
        return {"bytes": 2 * el * n, "flops": 0}
    if k == "krylov":
        return {"bytes": 3 * el * size["v"], "flops": 3 * mul * size["v"]}
    n = sum(d[0] * d[0] * d[1] for b in _layout(sym, shapes["X"])[0].values() for _, d, _ in b[3])
    return {"bytes": el * (n + sum(d * d for d in shapes["X"][0][0][0].values())), "flops": n}


# ---- exact values ---------------------------------------------------------------------------------
def _axes(leg):
    """First dense index of every stored key (U(1): one-dimensional irreps)."""
    out, o = {}, 0
    for s in sorted(leg[0], key=lambda s: _key("U1", s)):
        out[s] = o
        o += leg[0][s]
    return out, o


def _dense_views(W, x, dense):
    """Pairs (sub-block of the flat vector x, its place in the dense array) of a U(1) tensor."""
    legs = list(W[0]) + list(W[1])
    axes = [_axes(leg) for leg in legs]
    for b in _layout("U1", W)[0].values():
        for r in b[3]:
            for q in b[4]:
                at = []
                for leg, (first, _), s, d in zip(legs, axes, r[0] + q[0], r[1] + q[1]):
                    o = first[_dual("U1", s) if leg[1] else s]
                    at.append(slice(o, o + d))
                yield _sub(x, b, r, q), tuple(at)


def _to_dense(W, x):
    out = torch.zeros([_axes(leg)[1] for leg in list(W[0]) + list(W[1])], dtype=x.dtype, device=x.device)
    for sub, at in _dense_views(W, x, out):
        out[at] = sub
    return out


def _from_dense(W, dense):
    x = torch.zeros(_layout("U1", W)[1], dtype=dense.dtype, device=dense.device)
    for sub, at in _dense_views(W, x, dense):
        sub.copy_(dense[at])
    return x


def _apply_left(sym, shape_a, A, shape_e, E, adjoint=False):
    """(E ⊗ 1)·A for A in V⊗P ← V and E in V ← V."""
    out = torch.zeros_like(A)
    lay_a, lay_e = _layout(sym, shape_a)[0], _layout(sym, shape_e)[0]
    for b in lay_a.values():
        blk, res = _block(A, b), _block(out, b)
        for secs, degs, r0 in b[3]:
            if secs[0] not in lay_e:
                continue
            e = _block(E, lay_e[secs[0]])
            e = e.conj().T if adjoint else e
            rows = blk[r0:r0 + _prod(degs)].reshape(degs[1], degs[0], -1)  # the first leg is fastest
            res[r0:r0 + _prod(degs)] = torch.matmul(e, rows).reshape(_prod(degs), -1)
    return out


def _exact_env(sym, shapes, d):
    M = _apply_left(sym, shapes["A"], d["A"], shapes["E"], d["E"])
    lay_e, n = _layout(sym, shapes["E"])
    out = torch.zeros(n, dtype=M.dtype, device=M.device)
    for c, b in _layout(sym, shapes["A"])[0].items():
        _block(out, lay_e[c]).copy_(_block(d["A"], b).conj().T @ _block(M, b))
    return out


def _exact_grad(sym, shapes, d):
    A = d["A"]
    lay_a, lay_e = _layout(sym, shapes["A"])[0], _layout(sym, shapes["EL"])[0]
    M = _apply_left(sym, shapes["A"], A, shapes["EL"], d["EL"])
    N = _apply_left(sym, shapes["A"], A, shapes["EL"], d["EL"], adjoint=True)
    f = torch.zeros(1, dtype=A.dtype, device=A.device)
    dA, dEL, dER = torch.zeros_like(A), torch.zeros_like(d["EL"]), torch.zeros_like(d["ER"])
    for c, b in lay_a.items():
        ab, mb, nb = _block(A, b), _block(M, b), _block(N, b)
        er = _block(d["ER"], lay_e[c])
        g = ab.conj().T @ mb
        f += _dim(sym, c) * torch.trace(g @ er)
        _block(dA, b).copy_(mb @ er + nb @ er.conj().T)
        _block(dER, lay_e[c]).copy_(g.conj().T)
        for secs, degs, r0 in b[3]:
            if secs[0] in lay_e:
                a = ab[r0:r0 + degs[0]]  # the physical leg has one state per sector
                w = _dim(sym, c) / _dim(sym, secs[0])
                _block(dEL, lay_e[secs[0]]).add_((a @ er @ a.conj().T).conj().T, alpha=w)
    return [f, dA, dEL, dER]


@lru_cache(maxsize=None)
def _cg(a, b, c):
    """Clebsch-Gordan coefficients <a m1 b m2 | c m3> (twice-spins; m = j, j-1, ..., -j) by the
    Racah formula on exact integers."""
    f = math.factorial
    h = lambda x: x // 2  # noqa: E731
    out = np.zeros((a + 1, b + 1, c + 1))
    for i in range(a + 1):
        for j in range(b + 1):
            m1, m2 = a - 2 * i, b - 2 * j
            m3 = m1 + m2
            if abs(m3) > c:
                continue
            pre = (c + 1) * f(h(c + a - b)) * f(h(c - a + b)) * f(h(a + b - c)) / f(h(a + b + c) + 1)
            pre *= f(h(c + m3)) * f(h(c - m3)) * f(h(a - m1)) * f(h(a + m1)) * f(h(b - m2)) * f(h(b + m2))
            s = 0.0
            for k in range(0, h(a + b - c) + 1):
                den = [k, h(a + b - c) - k, h(a - m1) - k, h(b + m2) - k, h(c - b + m1) + k, h(c - a - m2) + k]
                if min(den) >= 0:
                    s += (-1) ** k / _prod(f(x) for x in den)
            out[i, j, (c - m3) // 2] = math.sqrt(pre) * s
    return out


def _bend(j):
    """The isomorphism of a dual leg: sqrt(2j+1) <j m1 j m2 | 0 0>."""
    return math.sqrt(j + 1) * _cg(j, j, 0)[:, :, 0]


def _exact_recouple(shapes, x):
    V = shapes["T"][0][0]
    src, _ = _layout("SU2", shapes["T"])
    dual = (V[0], True)
    dst, n = _layout("SU2", ((V, dual), (dual, V)))
    out = torch.zeros(n, dtype=x.dtype, device=x.device)
    src_rows = {c: {r[0]: r for r in b[3]} for c, b in src.items()}
    dst_rows = {c: {r[0]: r for r in b[3]} for c, b in dst.items()}
    spins = [s[0] for s in V[0]]
    for a in spins:
        for b in spins:
            for c in spins:
                for d in spins:
                    ks = [k for k in range(abs(a - b), a + b + 1, 2) if abs(c - d) <= k <= c + d and (c + d - k) % 2 == 0]
                    ls = [k for k in range(abs(a - c), a + c + 1, 2) if abs(b - d) <= k <= b + d and (b + d - k) % 2 == 0]
                    if not ks:
                        continue
                    F = {k: np.einsum("abm,cdm->acbd", _cg(a, b, k), _cg(c, d, k)) for k in ks}
                    subs = {k: _sub(x, src[(k,)], src_rows[(k,)][((a,), (b,))], src_rows[(k,)][((c,), (d,))]).permute(0, 2, 1, 3)
                            for k in ks}
                    for l in ls:
                        G = np.einsum("cq,aqm,bp,pdm->acbd", _bend(c), _cg(a, c, l), _bend(b), _cg(b, d, l))
                        to = _sub(out, dst[(l,)], dst_rows[(l,)][((a,), (c,))], dst_rows[(l,)][((b,), (d,))])
                        for k in ks:
                            u = float((G * F[k]).sum()) / (l + 1)
                            if abs(u) > 1e-14:
                                to.add_(subs[k], alpha=u)
    return out


def exact(case, seed):
    sym, shapes = _shapes(case)
    d = _inputs(case, seed)
    k = case["kind"]
    if k == "pair":
        (V, P), _ = shapes["A"]
        A, B = (_to_dense(shapes[n], d[n]) for n in ("A", "B"))
        C = torch.einsum("apc,cqb->apqb", A, B)
        dual = (P[0], True)
        return [_from_dense(((V, P, P), (V,)), C),
                _from_dense(((V, P), (dual, V)), C.permute(0, 2, 1, 3))]
    if k == "env":
        return _exact_env(sym, shapes, d)
    if k == "heff":
        t = {n: _to_dense(shapes[n], d[n]) for n in shapes}
        y = torch.einsum("awc,crsd->awrsd", t["L"], t["x"])
        y = torch.einsum("awrsd,wprv->asdpv", y, t["W1"])
        y = torch.einsum("asdpv,vqsu->adpqu", y, t["W2"])
        return _from_dense(shapes["x"], torch.einsum("adpqu,dub->apqb", y, t["R"]))
    if k == "grad":
        return _exact_grad(sym, shapes, d)
    if k == "recouple":
        return _exact_recouple(shapes, d["T"])
    if k == "regroup":
        (V, P, _), _ = shapes["x"]
        Vd, Pd = (V[0], True), (P[0], True)
        dense = _to_dense(shapes["x"], d["x"])
        if case["adjoint"]:
            return _from_dense(((Vd, Pd), (P, Vd)), dense.conj())
        return _from_dense(((V, P), (V, Pd)), dense.permute(0, 1, 3, 2))
    if k == "krylov":
        weight = torch.zeros_like(d["v"].real)
        for c, b in _layout(sym, shapes["v"])[0].items():
            weight[b[0]:b[0] + b[1] * b[2]] = _dim(sym, c)
        a = (weight * d["v"].conj() * d["w"]).sum()
        z = d["w"] - a * d["v"]
        n = (weight * (z.conj() * z).real).sum().sqrt()
        return [float(a.real), float(a.imag) if a.is_complex() else 0.0, float(n), z / n]
    (V, _), _ = shapes["X"]
    lay_v, n = _layout(sym, ((V,), (V,)))
    out = torch.zeros(n, dtype=d["X"].dtype, device=d["X"].device)
    for c, b in _layout(sym, shapes["X"])[0].items():
        for r in b[3]:
            t = _sub(d["X"], b, r, (r[0], r[1], r[2])).diagonal(dim1=1, dim2=3).sum(-1)
            _block(out, lay_v[r[0][0]]).add_(t, alpha=_dim(sym, c) / _dim(sym, r[0][0]))
    return out

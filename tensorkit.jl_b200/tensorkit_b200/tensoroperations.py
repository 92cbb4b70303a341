"""TensorOperations backend interface on device tensors, and the `@tensor` lowering.

Follows `src/tensors/tensoroperations.jl`:
- `tensoradd!` (`:44-62`): conj handled through the lazy adjoint and `adjointtensorindices`;
- `tensorcontract!` (`:130-161`) → `contract!` (`:318-357`), which evaluates the four index
  orders of `_contract_candidates` (`:360-376`) with `_contract_memcost` (`:378-383`) and
  calls `blas_contract!` (`:392-462`): permute A and B into (open; contracted) form unless
  they already are, blockwise `mul!`, permute C back unless it is a BLAS destination;
- `tensoradd_structure` / `tensorcontract_structure` (`:72-81`, `:174-182`).

Index tuples are 1-based (p = (p₁, p₂)), exactly as in TensorKit.

`tensor(expr, **tensors)` lowers an `@tensor` expression
(`"C[a,p,q;b] := A[a,p;c]*B[c,q;b]"`, factors optionally wrapped in `conj(...)`) into
pairwise `tensorcontract!` calls from left to right, as TensorOperations' `@tensor` does
without an explicit contraction order. Intermediates keep (open legs of the left operand ;
open legs of the right operand) as (codomain ; domain), which makes them BLAS
destinations of the blockwise `mul!`.
"""
from __future__ import annotations

import re
from functools import lru_cache

from . import _lib as L
from . import backend
from . import indexmanipulations as _im
from . import linalg as _la
from .backend import get_context, precision
from .indexmanipulations import (_ONE, _ZERO, _braid_table, _check_device, _current_stream, _scalar, dtype_code,
                                 permute, permute_)
from .linalg import gemm_plan, mul_
from .spaces import HomSpace, SpaceMismatch
from .tensor import AbstractTensorMap, AdjointTensorMap, TensorMap, new_tensor

__all__ = ["tensoradd_", "tensorcontract_", "tensorcontract", "contract_", "blas_contract_",
           "tensortrace_", "tensortrace", "tensortrace_structure",
           "tensoradd_structure", "tensorcontract_structure", "tensor", "parse_tensor_expr",
           "adjointtensorindices"]


# ---- index helpers ------------------------------------------------------------------
def adjointtensorindex(t, i):
    return t.numin() + i if i <= t.numout() else i - t.numout()


def adjointtensorindices(t, p):
    if len(p) == 2 and isinstance(p[0], tuple):
        return (tuple(adjointtensorindex(t, i) for i in p[0]),
                tuple(adjointtensorindex(t, i) for i in p[1]))
    return tuple(adjointtensorindex(t, i) for i in p)


def _linearize(p):
    return tuple(p[0]) + tuple(p[1])


def _canonicalize(p, t):
    if len(p[0]) == t.numout() and len(p[1]) == t.numin():
        return (tuple(p[0]), tuple(p[1]))
    lin = _linearize(p)
    return (lin[:t.numout()], lin[t.numout():])


def _invperm(p):
    out = [0] * len(p)
    for i, x in enumerate(p):
        out[x - 1] = i + 1
    return tuple(out)


def _repartition(p, n1):
    return (tuple(p[:n1]), tuple(p[n1:]))


def _oindABinC(pAB, pA, pB):
    return _repartition(_invperm(_linearize(pAB)), len(pA[0]))


def _adjoint(t):
    return t.parent if isinstance(t, AdjointTensorMap) else AdjointTensorMap(t)


# ---- structures -----------------------------------------------------------------------
def tensoradd_structure(A, pA, conjA=False) -> HomSpace:
    if not conjA:
        return A.space.select(pA)
    return tensoradd_structure(_adjoint(A), adjointtensorindices(A, pA), False)


def tensorcontract_structure(A, pA, conjA, B, pB, conjB, pAB) -> HomSpace:
    sA = tensoradd_structure(A, pA, conjA)
    sB = tensoradd_structure(B, pB, conjB)
    return sA.compose(sB).permute(pAB)


# ---- tensoradd! -------------------------------------------------------------------------
def tensoradd_(C, A, pA, conjA, alpha=1.0, beta=0.0):
    if conjA:
        Ap = _adjoint(A)
        pAp = adjointtensorindices(A, _canonicalize(pA, C))
        return permute_(C, Ap, pAp, alpha, beta)
    return permute_(C, A, _canonicalize(pA, C), alpha, beta)


# ---- contraction --------------------------------------------------------------------------
def has_shared_permute(t, p):
    p = (tuple(p[0]), tuple(p[1]))
    if isinstance(t, AdjointTensorMap):
        q = (adjointtensorindices(t, p[1]), adjointtensorindices(t, p[0]))
        return has_shared_permute(t.parent, q)
    return p == (t.codomainind(), t.domainind())


def _isblas(t, p):
    return has_shared_permute(t, p)


def _contract_candidates(pA, pB, pAB):
    N1, N2 = len(pA[0]), len(pB[1])
    qA = sorted(range(len(pA[1])), key=lambda i: pA[1][i])
    pA1 = (pA[0], tuple(pA[1][i] for i in qA))
    pB1 = (tuple(pB[0][i] for i in qA), pB[1])
    qB = sorted(range(len(pB[0])), key=lambda i: pB[0][i])
    pA2 = (pA[0], tuple(pA[1][i] for i in qB))
    pB2 = (tuple(pB[0][i] for i in qB), pB[1])
    f = lambda n: n - N1 if n > N1 else n + N2
    pABp = (tuple(map(f, pAB[0])), tuple(map(f, pAB[1])))
    return pA1, pB1, pA2, pB2, pABp


def _memcost(dA, dB, dC, C, A, pA, B, pB, pAB):
    ipAB = _oindABinC(pAB, pA, pB)
    return (dA * (not _isblas(A, pA) or A.data.dtype != C.data.dtype)
            + dB * (not _isblas(B, pB) or B.data.dtype != C.data.dtype)
            + dC * (not _isblas(C, ipAB)))


def _dim(t):
    return t.space.dim() if not isinstance(t, AdjointTensorMap) else t.parent.space.dim()


def _choose_order(C, A, pA, B, pB, pAB):
    """The index order that moves the least data: (exchange A and B, pX, pY, pXY)."""
    if len(pA[1]) != len(pB[0]):
        raise IndexError("number of contracted indices does not match")
    pA1, pB1, pA2, pB2, pABp = _contract_candidates(pA, pB, pAB)
    dA, dB, dC = _dim(A), _dim(B), _dim(C)
    m1 = _memcost(dA, dB, dC, C, A, pA1, B, pB1, pAB)
    m2 = _memcost(dA, dB, dC, C, A, pA2, B, pB2, pAB)
    rv = lambda p: (p[1], p[0])
    m3 = _memcost(dB, dA, dC, C, B, rv(pB1), A, rv(pA1), pABp)
    m4 = _memcost(dB, dA, dC, C, B, rv(pB2), A, rv(pA2), pABp)
    if min(m1, m2) <= min(m3, m4):
        return (False, pA1, pB1, pAB) if m1 <= m2 else (False, pA2, pB2, pAB)
    if m3 <= m4:
        return True, rv(pB1), rv(pA1), pABp
    return True, rv(pB2), rv(pA2), pABp


def contract_(C, A, pA, B, pB, pAB, alpha=1.0, beta=0.0):
    swap, pX, pY, pXY = _choose_order(C, A, pA, B, pB, pAB)
    X, Y = (B, A) if swap else (A, B)
    return blas_contract_(C, X, pX, Y, pY, pXY, alpha, beta)


def _alloc(W, like):
    return new_tensor(W, like.data.dtype, like.data.device)


def blas_contract_(C, A, pA, B, pB, pAB, alpha=1.0, beta=0.0, plan_hook=None):
    copyA = not (_isblas(A, pA) and A.data.dtype == C.data.dtype)
    if copyA:
        Anew = _alloc(tensoradd_structure(A, pA, False), C)
        tensoradd_(Anew, A, pA, False, 1.0, 0.0)
    else:
        Anew = permute(A, pA)
    copyB = not (_isblas(B, pB) and B.data.dtype == C.data.dtype)
    if copyB:
        Bnew = _alloc(tensoradd_structure(B, pB, False), C)
        tensoradd_(Bnew, B, pB, False, 1.0, 0.0)
    else:
        Bnew = permute(B, pB)
    pAnew = (Anew.codomainind(), Anew.domainind())
    pBnew = (Bnew.codomainind(), Bnew.domainind())
    ipAB = _oindABinC(pAB, pAnew, pBnew)
    if not _isblas(C, ipAB):
        Cnew = _alloc(tensoradd_structure(C, ipAB, False), C)
        mul_(Cnew, Anew, Bnew, 1.0, 0.0)
        tensoradd_(C, Cnew, pAB, False, alpha, beta)
    else:
        Cnew = permute(C, ipAB)
        mul_(Cnew, Anew, Bnew, alpha, beta)
    return C


class _Shape(AbstractTensorMap):
    """What the lowering needs to know of a tensor that does not exist yet: space and scalar type."""

    class _Data:
        __slots__ = ("dtype",)

        def __init__(self, dtype):
            self.dtype = dtype

    def __init__(self, space, dtype):
        self.space = space
        self.data = _Shape._Data(dtype)


class _Recipe:
    """A contraction lowered once per structure: the space of the result, which operands are permuted
    first (with their device tables and spaces), the GEMM plan per precision setting, and the final
    permute. It holds no data. Tables and plans belong to the context's caches; a recipe whose entries
    were evicted there is made again."""
    __slots__ = ("W", "swap", "adj", "move", "wc", "move_c", "plans", "used")

    def usable(self):
        for m in self.move:
            if m is not None and m[1].handle is None:
                return False
        return self.move_c is None or self.move_c.handle is not None


def _make_recipe(ctx, A, pA, conjA, B, pB, conjB, pAB):
    r = _Recipe()
    dt = A.data.dtype
    r.W = tensorcontract_structure(A, pA, conjA, B, pB, conjB, pAB)
    r.adj = (bool(conjA), bool(conjB))
    if conjA:
        A, pA = _adjoint(A), adjointtensorindices(A, pA)
    if conjB:
        B, pB = _adjoint(B), adjointtensorindices(B, pB)
    C = _Shape(r.W, dt)
    r.swap, pX, pY, pXY = _choose_order(C, A, pA, B, pB, pAB)
    new, moves = [], []
    for t, p in ((B, pX), (A, pY)) if r.swap else ((A, pX), (B, pY)):
        if _isblas(t, p):
            new.append(t)
            moves.append(None)
        else:
            W = tensoradd_structure(t, p, False)
            conj = 1 if isinstance(t, AdjointTensorMap) and t.is_complex() else 0
            moves.append((W, _braid_table(ctx, W, t, p, range(1, t.numind() + 1)), conj))
            new.append(_Shape(W, dt))
    r.move = tuple(moves)
    X, Y = new
    ip = _oindABinC(pXY, (X.codomainind(), X.domainind()), (Y.codomainind(), Y.domainind()))
    r.wc = r.move_c = None
    if not _isblas(C, ip):
        r.wc = tensoradd_structure(C, ip, False)
        t = _Shape(r.wc, dt)
        r.move_c = _braid_table(ctx, r.W, t, pXY, range(1, t.numind() + 1))
    r.plans = {}
    r.used = False
    return r


def _recipe(A, pA, conjA, B, pB, conjB, pAB):
    """The recipe of a contraction, or None where the step-by-step path has to run (operands that it
    refuses, launches that are being recorded)."""
    a, b = A.data, B.data
    dev = a.get_device()
    if dev != b.get_device():
        _check_device(A, B)
    if dev < 0 or a.dtype != b.dtype or _im.LAUNCH_LOG is not None or _la.FLOP_LOG is not None:
        return None, None
    ctx = get_context(dev)
    key = (A.space, type(A), pA, conjA, B.space, type(B), pB, conjB, pAB, a.dtype)
    r = ctx.recipes.get(key)
    if r is None or not r.usable():
        r = _make_recipe(ctx, A, pA, conjA, B, pB, conjB, pAB)
        ctx.recipes.pop(key, None)
        ctx.recipes.get_or(key, lambda: r)
    r.used = True
    return ctx, r


def _run_recipe(ctx, r, C, A, B, alpha, beta, keep):
    """Enqueue a lowered contraction. The library stream is ordered after and before the caller's once
    for all launches. The permuted operands are allocated on the caller's stream before the first (the
    memory may have been in use by work that another thread enqueued there a moment ago) and released
    after the second, so it is reused neither way too early. `keep`: C was passed in (its memory may
    belong to another stream's pool)."""
    lib, h = ctx.lib, ctx.handle
    out = C.data
    dtype, device = out.dtype, out.device
    code = dtype_code(out)
    if r.adj[0]:
        A = _adjoint(A)
    if r.adj[1]:
        B = _adjoint(B)
    ops = [B, A] if r.swap else [A, B]
    moved = [None if m is None else new_tensor(m[0], dtype, device) for m in r.move]
    D = C if r.move_c is None else new_tensor(r.wc, dtype, device)
    cur = _current_stream(ctx)
    joined = cur != ctx.stream_handle
    rc = lib.tkb_ctx_after(h, cur) if joined else 0
    if rc:
        L.check(rc, h)
    try:
        for i, m in enumerate(r.move):
            if m is not None:
                t = moved[i]
                m[1].used = True
                rc = lib.tkb_treetransform(h, m[1].handle, code, t.data.data_ptr(), ops[i].data.data_ptr(), _ONE,
                                           _ZERO, m[2])
                if rc:
                    L.check(rc, h)
                ops[i] = t
        X, Y = ops
        mode = precision()
        plan = r.plans.get(mode)
        if plan is None or plan.handle is None:
            plan = gemm_plan(ctx, D, X, Y)
            if len(r.plans) >= 16:
                r.plans.clear()
            r.plans[mode] = plan
        plan.used = True
        al = _ONE if alpha == 1.0 else _scalar(alpha)
        be = _ZERO if beta == 0.0 else _scalar(beta)
        if r.move_c is None:
            rc = lib.tkb_grouped_gemm(h, plan.handle, out.data_ptr(), X.data.data_ptr(), Y.data.data_ptr(), al, be)
        else:
            r.move_c.used = True
            rc = lib.tkb_grouped_gemm(h, plan.handle, D.data.data_ptr(), X.data.data_ptr(), Y.data.data_ptr(), _ONE,
                                      _ZERO)
            if rc == 0:
                rc = lib.tkb_treetransform(h, r.move_c.handle, code, out.data_ptr(), D.data.data_ptr(), al, be, 0)
        if rc:
            L.check(rc, h)
        if backend.USE_LOG is not None:
            backend.USE_LOG += [m[1] for m in r.move if m is not None] + [plan]
            if r.move_c is not None:
                backend.USE_LOG.append(r.move_c)
    finally:
        if joined:
            rc = lib.tkb_ctx_before(h, cur)
            if keep:
                out.record_stream(ctx.stream)
            if rc:
                L.check(rc, h)
    return C


def _pair(p):
    return (tuple(p[0]), tuple(p[1]))


def tensorcontract_(C, A, pA, conjA, B, pB, conjB, pAB, alpha=1.0, beta=0.0):
    pA, pB = _pair(pA), _pair(pB)
    pABc = _canonicalize(pAB, C)
    ctx, r = _recipe(A, pA, conjA, B, pB, conjB, pABc)
    W = r.W if r is not None else tensorcontract_structure(A, pA, conjA, B, pB, conjB, pABc)
    if W != C.space:
        raise SpaceMismatch(f"incompatible spaces for tensorcontract: {W} ≠ {C.space}")
    if C.data.get_device() != A.data.get_device():
        _check_device(C, A)
    if r is not None and C.data.dtype == A.data.dtype:
        return _run_recipe(ctx, r, C, A, B, alpha, beta, True)
    if conjA:
        A, pA = _adjoint(A), adjointtensorindices(A, pA)
    if conjB:
        B, pB = _adjoint(B), adjointtensorindices(B, pB)
    return contract_(C, A, pA, B, pB, pABc, alpha, beta)


def tensorcontract(A, pA, conjA, B, pB, conjB, pAB, alpha=1.0):
    pA, pB, pAB = _pair(pA), _pair(pB), _pair(pAB)
    ctx, r = _recipe(A, pA, conjA, B, pB, conjB, pAB)
    if r is not None:
        return _run_recipe(ctx, r, _alloc(r.W, A), A, B, alpha, 0.0, False)
    W = tensorcontract_structure(A, pA, conjA, B, pB, conjB, pAB)
    C = _alloc(W, A)
    return tensorcontract_(C, A, pA, conjA, B, pB, conjB, pAB, alpha, 0.0)


# ---- @tensor -------------------------------------------------------------------------------
_TERM = re.compile(r"\s*(conj\()?\s*([A-Za-z_][A-Za-z_0-9′']*)\s*\[([^\]]*)\]\s*(\))?\s*")


def _labels(s):
    if ";" in s:
        a, b = s.split(";", 1)
    else:
        a, b = s, ""
    sp = lambda x: tuple(y.strip() for y in x.split(",") if y.strip())
    return sp(a), sp(b)


def parse_tensor_expr(expr):
    """Parse 'C[a;b] := A[a;c]*conj(B[c;b])' → (lhs_name, (cod, dom), op, [(name, labels, conj)])."""
    lhs_name, lhs, op, factors = _parsed(expr)
    return lhs_name, lhs, op, list(factors)


@lru_cache(maxsize=1024)
def _parsed(expr):
    for op in (":=", "+=", "="):
        if op in expr:
            lhs, rhs = expr.split(op, 1)
            break
    else:
        raise ValueError("expression needs :=, = or +=")
    m = _TERM.fullmatch(lhs)
    if not m:
        raise ValueError(f"cannot parse left-hand side {lhs!r}")
    lhs_name = m.group(2)
    lcod, ldom = _labels(m.group(3))
    factors = []
    for part in rhs.split("*"):
        mm = _TERM.fullmatch(part)
        if not mm:
            raise ValueError(f"cannot parse factor {part!r}")
        conj = mm.group(1) is not None
        if conj != (mm.group(4) is not None):
            raise ValueError(f"unbalanced conj in {part!r}")
        c, d = _labels(mm.group(3))
        factors.append((mm.group(2), c + d, conj))
    return lhs_name, (lcod, ldom), op, tuple(factors)


def tensortrace_structure(A, p, conjA=False) -> HomSpace:
    """Space of the traced result: select(space(op(A)), p), the structure of tensoradd!
    (`src/tensors/tensoroperations.jl:72-81`, also used when indices are traced)."""
    return tensoradd_structure(A, p, conjA)


def tensortrace_(C, A, p, q, conjA=False, alpha=1.0, beta=0.0):
    """TO.tensortrace!(C, A, p, q, conjA, α, β) (`src/tensors/tensoroperations.jl:83-98`):
    conj(A) through the lazy adjoint with `adjointtensorindices`, then `trace_permute!`."""
    from .trace import trace_permute_
    if conjA:
        Ap = _adjoint(A)
        p2 = adjointtensorindices(A, _canonicalize(p, C))
        q2 = adjointtensorindices(A, q)
        return trace_permute_(C, Ap, p2, q2, alpha, beta)
    return trace_permute_(C, A, _canonicalize(p, C), q, alpha, beta)


def tensortrace(A, p, q, conjA=False, alpha=1.0):
    """New tensor α·tensortrace(op(A), p, q)."""
    C = _alloc(tensortrace_structure(A, p, conjA), A)
    return tensortrace_(C, A, p, q, conjA, alpha, 0.0)


def _pairwise_steps(lhs, factors):
    """Plan of pairwise contractions: list of (labelsA, conjA, labelsB, conjB, pA, pB, pAB,
    out_labels, is_final)."""
    return list(_steps((tuple(lhs[0]), tuple(lhs[1])), tuple((n, tuple(lab), cj) for n, lab, cj in factors)))


@lru_cache(maxsize=1024)
def _steps(lhs, factors):
    steps = []
    cur_labels, cur_conj = factors[0][1], factors[0][2]
    n = len(factors)
    for idx in range(1, n):
        lb, cb = factors[idx][1], factors[idx][2]
        for lab in set(cur_labels):
            if cur_labels.count(lab) > 1:
                raise NotImplementedError("traces inside @tensor are not supported")
        contracted = [l for l in cur_labels if l in lb]
        openA = [l for l in cur_labels if l not in lb]
        openB = [l for l in lb if l not in cur_labels]
        pA = (tuple(cur_labels.index(l) + 1 for l in openA), tuple(cur_labels.index(l) + 1 for l in contracted))
        pB = (tuple(lb.index(l) + 1 for l in contracted), tuple(lb.index(l) + 1 for l in openB))
        out = openA + openB
        final = idx == n - 1
        if final:
            lcod, ldom = lhs
            if sorted(lcod + ldom) != sorted(out):
                raise ValueError(f"left-hand side labels {lcod + ldom} ≠ open labels {out}")
            pAB = (tuple(out.index(l) + 1 for l in lcod), tuple(out.index(l) + 1 for l in ldom))
        else:
            pAB = (tuple(range(1, len(openA) + 1)), tuple(range(len(openA) + 1, len(out) + 1)))
        steps.append((cur_labels, cur_conj, lb, cb, pA, pB, pAB, tuple(out), final))
        cur_labels, cur_conj = tuple(out), False
    return steps


@lru_cache(maxsize=1024)
def _trace_labels(labels):
    """Leg pairs (q₁, q₂) of the labels repeated within one factor (1-based)."""
    reps = [l for l in dict.fromkeys(labels) if labels.count(l) > 1]
    for l in reps:
        if labels.count(l) > 2:
            raise ValueError(f"label {l!r} appears more than twice in one factor")
    q1 = tuple(labels.index(l) + 1 for l in reps)
    q2 = tuple(len(labels) - labels[::-1].index(l) for l in reps)
    return reps, (q1, q2)


def _pretrace(A, labels, conj):
    """Trace the labels a factor repeats (TensorOperations traces a factor before it enters
    a contraction); returns the traced tensor and its remaining labels."""
    labels = tuple(labels)
    reps, q = _trace_labels(labels)
    if not reps:
        return A, labels, conj
    nout = A.numout()
    keep = [i for i, l in enumerate(labels) if l not in reps]
    p = (tuple(i + 1 for i in keep if i < nout), tuple(i + 1 for i in keep if i >= nout))
    return tensortrace(A, p, q, conj), tuple(labels[i] for i in keep), False


def tensor(expr, out=None, alpha=1.0, **tensors):
    """Evaluate an @tensor expression on device TensorMaps.

    `:=` allocates the result; `=` writes into `out` (β = 0); `+=` accumulates (β = 1).
    Labels repeated within one factor are traced (`tensortrace!`)."""
    lhs_name, lhs, op, factors = parse_tensor_expr(expr)
    if len(factors) == 1:
        name, labels, conj = factors[0]
        A = tensors[name]
        lcod, ldom = lhs
        pA = (tuple(labels.index(l) + 1 for l in lcod), tuple(labels.index(l) + 1 for l in ldom))
        beta = 1.0 if op == "+=" else 0.0
        reps, q = _trace_labels(tuple(labels))
        if out is None:
            out = _alloc(tensoradd_structure(A, pA, conj), A)
        if reps:
            return tensortrace_(out, A, pA, q, conj, alpha, beta)
        return tensoradd_(out, A, pA, conj, alpha, beta)
    pre = [_pretrace(tensors[n], lab, cj) for n, lab, cj in factors]
    factors = [(n, lab, cj) for (n, _, _), (_, lab, cj) in zip(factors, pre)]
    steps = _pairwise_steps(lhs, factors)
    cur = pre[0][0]
    for i, (la, ca, lb, cb, pA, pB, pAB, outl, final) in enumerate(steps):
        B = pre[i + 1][0]
        if final:
            if out is None:
                if op != ":=":
                    raise ValueError("'=' and '+=' need an existing output tensor")
                return tensorcontract(cur, pA, ca, B, pB, cb, pAB, alpha)
            tensorcontract_(out, cur, pA, ca, B, pB, cb, pAB, alpha, 1.0 if op == "+=" else 0.0)
            return out
        cur = tensorcontract(cur, pA, ca, B, pB, cb, pAB, 1.0)
    raise AssertionError("unreachable")

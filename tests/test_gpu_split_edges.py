"""Edge cases of split precision in plans large enough to be sliced with the slice count left to the library (8 MFLOP
and more): every test asserts through the plan that the slices ran. Tolerance 1e-12, as in the other split tests.

Both forms of a slicing task are covered: rows contiguous in memory (op(A) = A, op(B) = B') and K contiguous (op(A) = A',
op(B) = B)."""
import numpy as np
import pytest

from helpers import O, cfg2_spaces, relerr, to_device, to_hom
import tensorkit_b200 as tk
from tensorkit_b200.linalg import gemm_plan

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _sliced(Cd, X, Y):
    plan = gemm_plan(tk.get_context(Cd.data.device.index), Cd, X, Y, "split")
    slices, fp64_tiles = plan.last_slices()
    assert plan.flops >= 8e6
    return slices, fp64_tiles


def _mul(X, Y, W, alpha=1.0, beta=0.0, C0=None):
    Cd = to_device(C0) if C0 is not None else tk.TensorMap.zeros(to_hom(W), dtype=X.data.dtype, device="cuda")
    tk.mul_(Cd, X, Y, alpha, beta, prec="split")
    return Cd, _sliced(Cd, X, Y)


def _dev(mat, adj):
    """A device tensor (or lazy adjoint of one) of one sector with this matrix."""
    sp = lambda d: O.Space({O.U1(0): d})  # noqa: E731
    stored = mat.conj().T if adj else mat
    t = O.BT(O.Hom([sp(stored.shape[0])], [sp(stored.shape[1])]), np.asfortranarray(stored).reshape(-1, order="F").copy())
    d = to_device(t)
    return tk.AdjointTensorMap(d) if adj else d


@pytest.mark.parametrize("adjA,adjB", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("cplx", [False, True])
def test_extreme_row_scales(cplx, adjA, adjB):
    """Rows of op(A) scaled by 1e-150 ... 1e150, a zero row, a row of subnormal values, columns of op(B) scaled by
    1e-100 ... 1e100: every entry keeps its accuracy relative to its row's and column's scale."""
    m, k, n = 200, 321, 150
    rng = np.random.default_rng(31)
    rnd = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s) if cplx else rng.standard_normal(s)  # noqa: E731
    a, b = rnd(m, k), rnd(k, n)
    a *= np.logspace(-150, 150, m)[:, None]
    a[5, :] = 0.0
    a[6, :] = rnd(k) * 1e-310  # subnormal row
    b *= np.logspace(-100, 100, n)[None, :]
    r = a @ b
    W = O.Hom([O.Space({O.U1(0): m})], [O.Space({O.U1(0): n})])
    Cd, (slices, _) = _mul(_dev(a, adjA), _dev(b, adjB), W)
    assert slices == [7]
    g = Cd.to_host().reshape(n, m).T
    # the error of an entry against |row max|·|column max|·K; scales below the normal range carry absolute
    # precision only, in the FP64 product as well
    scale = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :] * k
    normal = scale > 1e-290
    assert np.all(np.abs(g - r)[normal] <= TOL * scale[normal])
    assert np.all(np.abs(g - r)[~normal] <= 1e-300)
    assert np.all(g[5, :] == 0.0)
    assert np.count_nonzero(normal[6]) > 10


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("zero", ["A", "B"])
def test_zero_operand(cplx, zero):
    V, Pp = cfg2_spaces(4)
    A, B = O.randn(O.Hom([V, Pp], [V]), 4, cplx), O.randn(O.Hom([V], [V]), 5, cplx)
    (A if zero == "A" else B).data[:] = 0.0
    C0 = O.randn(O.mul(A, B).W, 6, cplx)
    Cd, (slices, _) = _mul(to_device(A), to_device(B), C0.W, 1.0, 0.5, C0)
    assert set(slices) == {7}  # and the check of the zero tiles, which no estimate passes, runs too
    assert relerr(Cd.to_host(), 0.5 * C0.data) <= 1e-15


@pytest.mark.parametrize("cplx", [False, True])
def test_products_and_adjoints(cplx):
    """C = A·B; C = α·A'·A + β·C with a lazy adjoint on the left, real and complex scalars; C = A·A'."""
    V, Pp = cfg2_spaces(4)
    A, B = O.randn(O.Hom([V, Pp], [V]), 1, cplx), O.randn(O.Hom([V], [V]), 2, cplx)
    Ad, Bd = to_device(A), to_device(B)
    ref = O.mul(A, B)
    Cd, (slices, _) = _mul(Ad, Bd, ref.W)
    assert 7 in slices and relerr(Cd.to_host(), ref.data) <= TOL
    ref = O.mul(A, A, adjA=True)
    C0 = O.randn(ref.W, 9, cplx)
    alpha, beta = (0.75 + 0.5j, -1.5 + 0.25j) if cplx else (0.75, -1.5)
    Cd, (slices, _) = _mul(tk.AdjointTensorMap(Ad), Ad, ref.W, alpha, beta, C0)
    assert 7 in slices and relerr(Cd.to_host(), alpha * ref.data + beta * C0.data) <= TOL
    ref = O.mul(A, A, adjB=True)
    Cd, (slices, _) = _mul(Ad, tk.AdjointTensorMap(Ad), ref.W)
    assert 7 in slices and relerr(Cd.to_host(), ref.data) <= TOL


@pytest.mark.parametrize("cplx", [False, True])
def test_missing_sectors_scale_by_beta(cplx):
    """Sectors of C that A·B does not reach get β·C, beside sectors that are sliced."""
    V = O.Space({O.U1(q): 130 for q in range(-2, 3)})
    V2 = O.Space({O.U1(q): 140 for q in range(0, 2)})
    A, B = O.randn(O.Hom([V], [V2]), 1, cplx), O.randn(O.Hom([V2], [V]), 2, cplx)
    ref = O.mul(A, B)
    C0 = O.randn(ref.W, 3, cplx)
    Cd, (slices, _) = _mul(to_device(A), to_device(B), ref.W, 2.0, 0.5, C0)
    assert sorted(slices) == [-1, -1, -1, 7, 7]
    assert relerr(Cd.to_host(), 2.0 * ref.data + 0.5 * C0.data) <= TOL


def test_small_environment_update_with_slices():
    """The smallest workload contraction, whose plans run in FP64 when the count is left open: seven slices asked for."""
    V, Pp = cfg2_spaces(1)
    A, E = O.randn(O.Hom([V, Pp], [V]), 1), O.randn(O.Hom([V], [V]), 1)
    fac = [("A", ("c", "p", "a"), True), ("E", ("c", "d"), False), ("A", ("d", "p", "b"), False)]
    ref = O.network(fac, (("a",), ("b",)), {"A": A, "E": E})
    with tk.using_precision("split", 7):
        got = tk.tensor("En[a;b] := conj(A[c,p;a])*E[c;d]*A[d,p;b]", A=to_device(A), E=to_device(E))
    ctx = tk.get_context(0)
    ran = [p.last_slices()[0] for k, p in ctx.plans.items() if k[0] == "gemm" and k[-2:] == ("split", 7)]
    assert any(7 in s for s in ran)
    assert relerr(got.to_host(), ref.data) <= TOL


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("adj", [False, True])
@pytest.mark.parametrize("m,k,n", [(200, 321, 150), (40, 7000, 33)])   # 7000: rows longer than a staged task's
@pytest.mark.parametrize("where", ["A", "B", "row of A"])
def test_nan_is_kept(cplx, adj, m, k, n, where):
    """One NaN, or a row of them, makes its row (column) of the product NaN and leaves the others as they are."""
    rng = np.random.default_rng(17)
    rnd = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s) if cplx else rng.standard_normal(s)  # noqa: E731
    a, b = rnd(m, k), rnd(k, n)
    want = a @ b
    if where == "B":
        b[k - 1, 5] = want[:, 5] = np.nan
    else:
        a[7, slice(None) if where != "A" else 3] = want[7, :] = np.nan
    W = O.Hom([O.Space({O.U1(0): m})], [O.Space({O.U1(0): n})])
    Cd, _ = _mul(_dev(a, adj), _dev(b, adj), W)
    got = Cd.to_host().reshape(n, m).T
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.abs(got - want)[ok].max() <= TOL * np.abs(want[ok]).max()

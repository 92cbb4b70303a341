"""Plain products whose speed must not hang on the form of the operands: a complex adjoint costs what its
materialised copy would."""
import pytest
import torch

import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu


def _best(fn, n=12):
    ctx, best = tk.get_context(0), 1e9
    with torch.cuda.stream(ctx.stream):
        for _ in range(3):
            fn()
        for _ in range(n):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(500_000)  # the calls are all enqueued before the first of them runs
            a.record()
            for _ in range(4):
                fn()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
    return best


def _hom(m, n):
    sp = lambda d: tk.ProductSpace([tk.Vect({tk.U1Irrep(0): d})])  # noqa: E731
    return tk.HomSpace(sp(m), sp(n))


def _rand(m, n, dtype):
    return tk.TensorMap(torch.randn(m * n, dtype=dtype, device="cuda"), _hom(m, n))


@pytest.mark.parametrize("side", ["A", "B"])
def test_complex_adjoint_costs_no_more(side):
    """At most a tenth more (measured 1.00; 1.19 with pieces of 16 bytes scattered in shared memory)."""
    m, k, n = 1500, 400, 1500
    A, B, C = (_rand(a, b, torch.complex128) for a, b in ((m, k), (k, n), (m, n)))
    adj = tk.AdjointTensorMap(_rand(k, m, torch.complex128) if side == "A" else _rand(n, k, torch.complex128))
    X, Y = (adj, B) if side == "A" else (A, adj)
    plain, other = _best(lambda: tk.mul_(C, A, B, prec="plain")), _best(lambda: tk.mul_(C, X, Y, prec="plain"))
    assert other <= 1.1 * plain


SHAPES = [(60, 2400, 2400), (2399, 1203, 61), (257, 1736, 400), (512, 100, 512), (1000, 20, 1000), (16, 16, 20000),
          (300, 301, 299), (5, 20000, 33)]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_values_of_uneven_shapes(m, k, n, cplx):
    """Both tile sizes, equal pieces of K and shares that end inside tiles, with alpha and beta, against torch."""
    dtype = torch.complex128 if cplx else torch.float64
    A, B, C = (_rand(a, b, dtype) for a, b in ((m, k), (k, n), (m, n)))
    mat = lambda t, r, c: t.data.view(c, r).t()  # noqa: E731
    want = 0.75 * (mat(A, m, k) @ mat(B, k, n)) - 0.5 * mat(C, m, n)
    tk.mul_(C, A, B, 0.75, -0.5, prec="plain")
    assert (mat(C, m, n) - want).abs().max() <= 1e-13 * k ** 0.5 * want.abs().max()  # a few u·sqrt(K)


@pytest.mark.parametrize("shape,of,cplx,ratio", [
    ((60, 2400, 2400), (1024, 1024, 1024), True, 0.44),    # of 0.32 of the work: measured 0.37, was 0.52
    ((60, 2400, 2400), (1024, 1024, 1024), False, 0.52),   # 0.47, was 0.56
    ((512, 100, 512), (512, 512, 512), False, 0.52)])      # of 0.2 of the work: 0.40, was 0.63
def test_uneven_shapes_keep_the_chip_busy(shape, of, cplx, ratio):
    dtype = torch.complex128 if cplx else torch.float64
    took = []
    for m, k, n in (shape, of):
        A, B, C = (_rand(a, b, dtype) for a, b in ((m, k), (k, n), (m, n)))
        took.append(_best(lambda: tk.mul_(C, A, B, prec="plain")))
    assert took[0] <= ratio * took[1]


def test_beta_costs_little_more_than_its_bytes():
    """A product of short K that adds to C: a fifth more time (36.3 us after 30.9; 41.4 when every column waited for
    its own old values)."""
    m, k, n = 2048, 64, 2048
    A, B, C = (_rand(a, b, torch.float64) for a, b in ((m, k), (k, n), (m, n)))
    plain, added = (_best(lambda: tk.mul_(C, A, B, 1e-3, beta, prec="plain")) for beta in (0.0, 0.5))
    assert added <= 1.28 * plain

"""The trace kernel's split of each sum over threads, at the sizes where the split changes: one
destination element (a full trace), fewer and more elements than a task holds, fewer terms than
slices, sums of several batches per thread, two and three traced pairs, α/β. U(1) coefficients are +1
and the data is shifted away from zero, so a sum of n ≤ 4096 terms is exact to n·2⁻⁵³ < 5e-13
relatively: bound 1e-12."""
import pytest

from helpers import O, U1, relerr, to_device
import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _sp(**degs):
    return O.Space({U1({"m": -1, "z": 0, "p": 1}[k]): d for k, d in degs.items()})


A, B, S, ONE = _sp(m=3, z=70, p=2), _sp(z=33, p=17), _sp(m=1, z=2), _sp(z=1)
LONG = _sp(z=1900, p=41)
CASES = {
    "full": (O.Hom([LONG], [LONG]), ((), ()), ((1,), (2,))),
    "full_two": (O.Hom([A, S], [A, S]), ((), ()), ((1, 2), (3, 4))),
    "few_elements": (O.Hom([S, B], [S, B]), ((1,), (3,)), ((2,), (4,))),
    "few_terms": (O.Hom([A, ONE], [B, ONE]), ((1,), (3,)), ((2,), (4,))),
    "ordinary": (O.Hom([A, S], [B, S]), ((1,), (3,)), ((2,), (4,))),
    "long_sums": (O.Hom([S, LONG], [LONG, S]), ((1,), (4,)), ((2,), (3,))),
    "three_pairs": (O.Hom([S, A, S, S], [A, S, S, S]), ((1,), (6,)), ((2, 3, 4), (5, 7, 8))),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("cplx", [False, True])
def test_trace_sums(name, cplx):
    W, p, q = CASES[name]
    t, d0 = O.randn(W, 5, cplx), O.randn(W.select(p), 6, cplx)
    t.data[:] = 4.0 + 0.5 * t.data
    out = tk.trace_permute(to_device(t), p, q)
    assert relerr(out.to_host(), O.trace_permute(t, p, q).data) <= TOL
    alpha, beta = (0.7 - 0.2j, -1.3 + 0.5j) if cplx else (0.7, -1.3)
    ref = O.trace_permute(t, p, q, alpha, tdst=d0, beta=beta)
    out = tk.trace_permute_(to_device(d0), to_device(t), p, q, alpha, beta)
    assert relerr(out.to_host(), ref.data) <= TOL

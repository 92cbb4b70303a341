"""Rounding of long sums in the plain products. Row [1, t, t, ...] with t = 2^-54 times a column of ones is
1 + (K - 1) t: a sum that holds the 1 loses every t that it takes one by one (half an ulp of 1 is 2 t), so
what the result lacks counts the products that met in one accumulator. Real 64x64 tiles keep a second one for
half of K; 32x32 tiles add whole stages of 16 (complex: four at a time). The final additions round once each (2 t)."""
import numpy as np
import pytest
import torch

import tensorkit_b200 as tk

pytestmark = pytest.mark.gpu
T = 2.0 ** -54


@pytest.mark.parametrize("cplx,m,k,together", [
    (False, 2048, 512, 256),      # 1024 tiles of 64x64, K uncut in most of them
    (False, 2047, 333, 173),      # odd: 8-byte copies, an incomplete last stage (8 of its positions in the first half)
    (False, 256, 128, 16), (False, 255, 97, 16), (False, 40, 16, 16),   # 32x32 tiles
    (True, 576, 576, 64), (True, 255, 97, 64)])
def test_no_accumulator_takes_all_of_k(cplx, m, k, together):
    sp = lambda d: tk.ProductSpace([tk.Vect({tk.U1Irrep(0): d})])  # noqa: E731
    one = 1 + 1j if cplx else 1.0   # imaginary parts run through the same sums
    a = np.full((m, k), T * one)
    a[:, 0] = one
    dtype = torch.complex128 if cplx else torch.float64
    A = tk.TensorMap(torch.from_numpy(a.ravel(order="F")).cuda(), tk.HomSpace(sp(m), sp(k)))
    B = tk.TensorMap(torch.ones(k * m, dtype=dtype, device="cuda"), tk.HomSpace(sp(k), sp(m)))
    got = torch.view_as_real(tk.compose(A, B).data) if cplx else tk.compose(A, B).data
    lost = 1.0 + (k - 1) * T - got.cpu().numpy()   # 1 + (k - 1) t itself is rounded by at most 2 t
    assert np.abs(lost).max() <= (together + 4) * T

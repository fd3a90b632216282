"""The FP32 operator of the refinement: at most 16 terms per FP32 sum, FP64
beyond, by the size of its error.

Each multiply-add of a chain is off by a uniform rounding of at most 2^-24 of
the partial sum, so a row's error has a variance of at most sum |partial|^2
2^-48 / 3 over its chains; the mantissas of the partial sums make it 0.54 of
that on average (RMS 0.74). The RMS over the rows of error / bound is held to
0.85; chains of 64 terms are beyond it at 20,011 columns (20 terms each there) and
have 1.9 at 40,000."""
import ctypes

import numpy as np
import pytest
import torch

from wavebem_gb300.bem_problem import load_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 1023, 1030, 3001, 20011, 40000])
def test_error_of_the_fp32_operator(n):
    L = load_library()
    L.wbem_test_matvec_s32.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] * 3
    ld = -(-n // 32) * 32
    gen = torch.Generator(device="cuda").manual_seed(n)
    S = torch.rand(n, ld, generator=gen, device="cuda", dtype=torch.float32)
    x = torch.rand(n, generator=gen, device="cuda", dtype=torch.float32).double()
    y = torch.empty(n, device="cuda", dtype=torch.float64)
    assert L.wbem_test_matvec_s32(n, ld, S.data_ptr(), x.data_ptr(), y.data_ptr()) == 0
    ratio = []
    for r in range(0, n, max(1, n // 400)):
        p = S[r, :n].double() * x
        err = float(y[r] - p.sum())
        q = torch.zeros(-(-n // 16384) * 16384, device="cuda", dtype=torch.float64)
        q[:n] = p
        part = q.view(-1, 16, 256, 4).cumsum(1)  # chains: columns 4 t + c + 1024 step, 16 steps
        var = float((part.square() * (q.view(-1, 16, 256, 4) != 0)).sum()) * 2.0 ** -48 / 3
        ratio.append(err / var ** 0.5)
    ratio = np.array(ratio)
    if n < 1000:  # a few rounding errors: each within its bound
        assert np.abs(ratio).max() <= 3 ** 0.5 * n ** 0.5
    else:
        assert np.sqrt(np.mean(ratio ** 2)) <= 0.85
    del S

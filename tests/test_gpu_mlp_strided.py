"""mmdg_mlp_gemm into a matrix whose rows are longer than the result (ldc > N): nothing but
its N columns is written, with K split over blocks (K >= 256 here) and without."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 255, 256, 1023, 1024, 8192])
@pytest.mark.parametrize("M,N,ldc", [(20, 12, 19), (1, 5, 8), (130, 64, 68), (53, 81, 200)])
def test_columns_past_n_and_memory_past_the_last_row_stay(M, N, ldc, K):
    import torch
    from mmd import _native
    from mmd.guess import DensityMLP
    L = _native.lib()
    DensityMLP._sig(L)
    g = torch.Generator(device="cuda").manual_seed(K)
    A, B = torch.randn(K, M, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    C = torch.full((M + 4, ldc), 7.0, device="cuda")  # four rows past the last one
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert L.mmdg_mlp_gemm(M, N, K, p(A), M, 1, 0, p(B), N, 0, 0, p(C), ldc, 0.0, _native.stream_ptr()) == 0
    ref = A.double().T @ B.double()
    # FP32 sums of K terms: relative 6e-8 sqrt(K) of their norm, ten times over
    assert float(torch.linalg.norm(C[:M, :N].double() - ref)) < (6e-7 * np.sqrt(K) + 1e-7) * float(torch.linalg.norm(ref))
    assert bool((C[:M, N:] == 7.0).all()) and bool((C[M:] == 7.0).all())

"""Coulomb and exchange from a stored tensor at the edges of the kernel's blocks, on tensors
and densities without any symmetry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 7, 16, 22, 23, 31, 33, 51, 64, 100])
def test_jk_dense_equals_einsum(N):
    import torch
    from mmd import _native
    rng = np.random.default_rng(N)
    T, P = rng.standard_normal((N,) * 4), rng.standard_normal((N, N))
    Td, Pd = torch.as_tensor(T, device="cuda"), torch.as_tensor(P, device="cuda")
    J, K = torch.full_like(Pd, np.nan), torch.full_like(Pd, np.nan)
    _native.scratch_context().jk_dense(Td, Pd, J, K)
    # N^2 products of unit normals, each summed with a relative rounding of 1.1e-16
    tol = 1.2e-16 * N * N * 12.0 + 1e-15
    assert np.abs(J.cpu().numpy() - np.einsum("pqrs,sr->pq", T, P)).max() < tol
    assert np.abs(K.cpu().numpy() - np.einsum("psqr,sr->pq", T, P)).max() < tol

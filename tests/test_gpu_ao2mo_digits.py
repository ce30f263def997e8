"""The AO -> MO transform on both sides of the tensor-core form's range and at the edges of
its tiles: tensors without symmetry whose rows span many decades, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _transform(T, C):
    x = T
    for _ in range(4):  # contract the first index, append the new one
        x = np.tensordot(x, C, axes=([0], [0]))
    return x


@pytest.mark.parametrize("N", [1, 2, 8, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 80])
def test_transform_equals_float64(N):
    import torch
    from mmd import _native
    rng = np.random.default_rng(N)
    T = rng.standard_normal((N,) * 4) * 10.0 ** rng.uniform(-9, 3, (N, N, N, 1))
    C = np.linalg.qr(rng.standard_normal((N, N)))[0] * 10.0 ** rng.uniform(-2, 2, N)
    out = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1))
    ref = _transform(T, C)
    got = out.cpu().numpy().reshape(ref.shape)
    # per quarter a rounding of 1.1e-16 and, in plain arithmetic, up to N of them in the sum:
    # 4 (1 + sqrt(N)) 1.1e-16 of the norm of each new-index slice, for both sides
    scale = np.linalg.norm(C, axis=0)
    err = np.linalg.norm((got - ref) / scale / scale[:, None] / scale[:, None, None] / scale[:, None, None, None])
    norm = np.linalg.norm(ref / scale / scale[:, None] / scale[:, None, None] / scale[:, None, None, None])
    assert err < 8 * (1 + np.sqrt(N)) * 1.1e-16 * norm


@pytest.mark.parametrize("N", [20, 40])
def test_non_finite_rows_and_columns(N):
    import torch
    from mmd import _native
    rng = np.random.default_rng(N)
    T = rng.standard_normal((N,) * 4)
    C = np.eye(N)  # one quarter at a time keeps what is finite apart
    T[3, 4, 5, 6] = np.inf
    out = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1))
    with np.errstate(invalid="ignore"):
        ref = _transform(T, C)
    got = out.cpu().numpy().reshape(ref.shape)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.isinf(got), np.isinf(ref))
    fine = np.isfinite(ref)
    assert np.abs(got[fine] - ref[fine]).max(initial=0.0) < 1e-14


@pytest.mark.parametrize("N", [18, 33])
def test_extreme_magnitudes(N):
    import torch
    from mmd import _native
    rng = np.random.default_rng(N)
    for scale in (1e-300, 1e-320, 1e290, 0.0):
        T = rng.standard_normal((N,) * 4) * scale
        C = np.linalg.qr(rng.standard_normal((N, N)))[0]
        out = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1))
        ref = _transform(T, C)
        got = out.cpu().numpy().reshape(ref.shape)
        # subnormal results: one unit (5e-324) per quarter and term
        assert np.abs(got - ref).max() <= 1e-14 * np.abs(ref).max() + 4 * N * 5e-324

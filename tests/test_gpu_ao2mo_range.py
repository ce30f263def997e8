"""The AO -> MO transform up to the end of the tensor-core form's range (N = 128), where its
integer sums come closest to 2^24, and past it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _transform(T, C):
    import torch
    for _ in range(4):  # contract the first index, append the new one
        T = torch.tensordot(T, C, dims=([0], [0]))
    return T


@pytest.mark.parametrize("N", [81, 96, 97, 112, 113, 127, 128, 129])
def test_transform_equals_float64(N):
    import torch
    from mmd import _native
    g = torch.Generator(device="cuda").manual_seed(N)
    T = torch.randn((N,) * 4, generator=g, device="cuda", dtype=torch.float64)
    C = torch.linalg.qr(torch.randn((N, N), generator=g, device="cuda", dtype=torch.float64).cpu())[0].cuda().contiguous()
    got = _native.ao2mo(C, T.reshape(-1)).view((N,) * 4)
    ref = _transform(T, C)
    # per quarter a rounding of 1.1e-16 and, in plain arithmetic, up to N of them in the sum:
    # 4 (1 + sqrt(N)) 1.1e-16 of the norm, for both sides
    assert float(torch.linalg.norm(got - ref)) < 8 * (1 + np.sqrt(N)) * 1.1e-16 * float(torch.linalg.norm(ref))


@pytest.mark.parametrize("N", [16, 127, 128])
def test_largest_digits_of_one_sign(N):
    import torch
    from mmd import _native
    # 2^62 - 128 (256^1 + ... + 256^6) in units of 2^-62: a top digit of 64, then six of -128
    v = (2 ** 62 - sum(128 << 8 * i for i in range(1, 7))) / 2.0 ** 62
    T = torch.full((N ** 4,), v, dtype=torch.float64, device="cuda")
    C = torch.full((N, N), v, dtype=torch.float64, device="cuda")
    got = _native.ao2mo(C, T)
    want = v * (N * v) ** 4
    # one rounding of 1.1e-16 per quarter, 5 in the expected value
    assert float((got - want).abs().max()) <= 9 * 1.2e-16 * want

"""Every element of the AO -> MO transform against the error bound of FP64 sums, on data whose
large elements meet small ones: the digits of the tensor-core form hold a row's and a column's
largest elements, so a sum without them needs another way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _transform(T, C):
    for _ in range(4):  # contract the first index, append the new one
        x = T.reshape(T.shape[0], -1)
        T = (x[:, :, None] * C[:, None, :]).sum(0).reshape(*T.shape[1:], C.shape[1])
    return T


def _check(T, C, ref, size):
    """Elementwise: a quarter transform's sum of N products is off by at most N 2^-53 of the sum
    of their magnitudes and rounded once, the four by four times that."""
    import torch
    from mmd import _native
    N = len(C)
    got = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1))
    err = np.abs(got.cpu().numpy().reshape((N,) * 4).astype(np.longdouble) - ref)
    assert (err <= 4 * (N + 1) * 2.0 ** -53 * size * (1 + 1e-10) + 4 * N * 5e-324).all(), float((err / size).max())


@pytest.mark.parametrize("g", [1e-3, 1e-6, 1e-8, 1e-12])
@pytest.mark.parametrize("N", [7, 16, 31, 64, 100])
def test_opposite_grading(N, g):
    """Rows and columns alternate between 1 and g in opposite positions, all terms positive."""
    rng = np.random.default_rng(N)
    t = rng.uniform(0.5, 1.0, (4, N)) * np.where(np.arange(N) % 2, g, 1.0)
    C = rng.uniform(0.5, 1.0, (N, N)) * np.where(np.arange(N) % 2, 1.0, g)[:, None]
    T = np.einsum("p,q,r,s->pqrs", *t)
    P, Q, R, S = ((x.astype(np.longdouble) @ C.astype(np.longdouble)) for x in t)
    ref = P[:, None, None, None] * Q[:, None, None] * R[:, None] * S
    # (T itself is a product rounded three times)
    import torch
    from mmd import _native
    got = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1))
    err = np.abs(got.cpu().numpy().reshape((N,) * 4).astype(np.longdouble) - ref)
    assert (err <= (4 * (N + 1) + 4) * 2.0 ** -53 * ref).all(), float((err / ref).max())


def _columns(kind, N, rng):
    if kind == "units":           # one element a column: a relabelling, exact in FP64
        return np.eye(N)[rng.permutation(N)]
    if kind == "blocks":          # symmetry-adapted or localised orbitals
        C = np.zeros((N, N))
        for b in np.array_split(np.arange(N), 3):
            C[np.ix_(b, b)] = np.linalg.qr(rng.standard_normal((len(b), len(b))))[0]
        return C
    return np.linalg.qr(rng.standard_normal((N, N)))[0] * 10.0 ** rng.uniform(-6, 0, (N, N))


@pytest.mark.parametrize("kind", ["units", "blocks", "graded"])
@pytest.mark.parametrize("N", [5, 16, 18])
@pytest.mark.parametrize("scale", [1.0, 1e-290, 1e200])
def test_decaying_rows(kind, N, scale):
    rng = np.random.default_rng(N)
    x = rng.uniform(0, 30, N)
    d = np.abs(x[:, None] - x[None, :])
    T = scale * rng.standard_normal((N,) * 4) * np.exp(-d[:, :, None, None] - d[None, None, :, :] - d[None, :, :, None])
    C = _columns(kind, N, rng)
    l = lambda a: a.astype(np.longdouble)
    _check(T, C, _transform(l(T), l(C)), _transform(np.abs(l(T)), np.abs(l(C))))


def test_zero_rows_and_columns():
    rng = np.random.default_rng(3)
    N = 33
    T, C = rng.standard_normal((N,) * 4), rng.standard_normal((N, N))
    T[:, :, 4] = 0.0
    T[7] = 0.0
    C[:, 5] = 0.0
    import torch
    from mmd import _native
    got = _native.ao2mo(torch.as_tensor(C, device="cuda"), torch.as_tensor(T, device="cuda").reshape(-1)).cpu().numpy()
    got = got.reshape((N,) * 4)
    for ax in range(4):
        assert not got.take(5, axis=ax).any()
    ref = np.einsum("pqrs,pP,qQ,rR,sS->PQRS", T, C, C, C, C, optimize=True)
    size = np.einsum("pqrs,pP,qQ,rR,sS->PQRS", *map(np.abs, (T, C, C, C, C)), optimize=True)
    # both sides round
    assert (np.abs(got - ref) <= 8 * (N + 1) * 2.0 ** -53 * size).all()

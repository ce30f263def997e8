"""The gradient of a class whose triangle of quartets passes 2^31: one group of 67,161 equal
pairs against the same functions written with two halves of a primitive, which spreads the
pairs over three groups."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(double, centre, exps, P, W):
    import torch
    from mmd import _native
    from mmd.integrals.shells import ShellSet
    n = len(exps)
    nprim = np.where(double, 2, 1).astype(np.int32)
    func = np.full((n, 6), -1, dtype=np.int32)
    func[:, 0] = np.arange(n)
    norm = (2 * exps / np.pi) ** 0.75
    ctx = _native.Context(ShellSet(n, np.zeros(n, dtype=np.int32), nprim, centre, np.repeat(exps, nprim),
                                   np.repeat(norm / nprim, nprim), func), prim_tol=0.0)
    natom = 3
    atom = (np.arange(n) % natom).astype(np.int32)
    xyz, Z = np.array([0.0, 0, 0, 0, 0, 9, 9, 0, 0]), np.ones(natom)
    grad = np.zeros(3 * natom)
    Pd, Wd = torch.as_tensor(P, device="cuda"), torch.as_tensor(W, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _native.check(_native.lib().mmdg_rhf_gradient(ctx._h, p(Pd), p(Wd), natom, _native._ptr(xyz), _native._ptr(Z),
                                                  _native._ptr(atom), 0.0, _native._ptr(grad), _native.stream_ptr()),
                  "mmdg_rhf_gradient")
    return grad


def test_triangle_of_65536_pairs_and_more():
    n = 366
    rng = np.random.default_rng(n)
    centre, exps = rng.uniform(0, 8, (n, 3)), rng.uniform(0.3, 1.0, n)
    P, W = (0.5 * (A + A.T) for A in rng.standard_normal((2, n, n)))
    one = _gradient(np.zeros(n, dtype=bool), centre, exps, P, W)
    two = _gradient(np.arange(n) >= n // 2, centre, exps, P, W)
    # 2.3e9 terms of random sign, each rounded by about 1e-16 of its size: a relative 1e-16
    # sqrt(2.3e9) = 5e-12 of the sum's own size, a hundred times over for the larger ones
    assert np.abs(one).max() > 0
    assert np.abs(one - two).max() < 5e-10 * np.abs(one).max()

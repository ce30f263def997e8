"""The guess network's fused layer kernels at the edges of their tiles against float64."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows,out,inp", [(1, 1, 1), (2, 81, 53), (127, 64, 16), (128, 65, 17), (129, 225, 256),
                                          (1025, 256, 53), (4099, 225, 33)])
def test_linear_back_and_weight_gradient(rows, out, inp):
    import torch
    from mmd import _native
    from mmd.guess import DensityMLP
    L = _native.lib()
    DensityMLP._sig(L)
    rng = np.random.default_rng(rows)
    f = lambda *s: torch.as_tensor(rng.standard_normal(s).astype(np.float32), device="cuda")
    X, b, dZ, Zp = f(rows, inp), f(out), f(rows, out), f(rows, inp)
    W = f(out, inp).to(torch.bfloat16)
    Z, Y = torch.empty(rows, out, device="cuda"), torch.empty(rows, out, device="cuda")
    dZp, db, dW = torch.empty(rows, inp, device="cuda"), torch.empty(inp, device="cuda"), torch.empty(out, inp, device="cuda")
    dbc = torch.empty(out, device="cuda")
    st = _native.stream_ptr()
    for silu in (0, 1):
        assert L.mmdg_mlp_linear(rows, out, inp, _p(X), _p(W), _p(b), _p(Z), _p(Y), silu, st) == 0
        assert L.mmdg_mlp_back(rows, out, inp, _p(dZ), _p(W), _p(Zp), _p(dZp), _p(db), silu, st) == 0
        z = X.double() @ W.double().T + b.double()
        y = torch.nn.functional.silu(z) if silu else z
        s = torch.sigmoid(Zp.double())
        d = (dZ.double() @ W.double()) * (s * (1 + Zp.double() * (1 - s)) if silu else 1.0)
        # FP32 sums of k terms: relative 6e-8 sqrt(k) of their norm, ten times over
        tol = lambda k: 6e-7 * np.sqrt(k) + 1e-7
        rel = lambda a, e: float(torch.linalg.norm(a.double() - e) / torch.linalg.norm(e))
        assert rel(Z, z) < tol(inp) and rel(Y, y) < tol(inp)
        assert rel(dZp, d) < tol(out) and rel(db, d.sum(0)) < tol(out) + tol(rows) * np.sqrt(rows)
    assert L.mmdg_mlp_gemm(out, inp, rows, _p(dZ), out, 1, 0, _p(X), inp, 0, 0, _p(dW), inp, 0.0, st) == 0
    assert L.mmdg_mlp_colsum(_p(dZ), _p(dbc), rows, out, st) == 0
    assert rel(dW, dZ.double().T @ X.double()) < tol(rows)
    assert rel(dbc, dZ.double().sum(0)) < tol(rows)
    M = (f(rows, out) > 0).float()
    T, dY = f(rows, out), torch.empty(rows, out, device="cuda")
    loss, count = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.empty(1, dtype=torch.float64, device="cuda")
    assert L.mmdg_mlp_mse_masked(_p(Y), _p(T), _p(M), _p(dY), _p(loss), _p(count), rows * out, st) == 0
    c = max(float(M.sum()), 1.0)
    e = (Y.double() - T.double()) * M.double()
    assert abs(float(loss) - float((e ** 2).sum()) / c) < 1e-6 * float((e ** 2).sum()) / c + 1e-12
    assert float(torch.linalg.norm(dY.double() - 2 * e / c)) < 1e-6 * float(torch.linalg.norm(2 * e / c)) + 1e-12


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 8192 * 81])
def test_loss_sums_32_neighbours_in_fp32(n):
    import torch
    from mmd import _native
    from mmd.guess import DensityMLP
    L = _native.lib()
    DensityMLP._sig(L)
    rng = np.random.default_rng(n)
    f = lambda: torch.as_tensor(rng.standard_normal(n).astype(np.float32), device="cuda")
    Y, T, M = f(), f(), (f() > 0).float()
    dY, loss = torch.empty_like(Y), torch.zeros(1, dtype=torch.float64, device="cuda")
    inv = np.float32(1.0 / max(float(M.sum()), 1.0))
    assert L.mmdg_mlp_mse(_p(Y), _p(T), _p(M), _p(dY), _p(loss), n, float(inv), _native.stream_ptr()) == 0
    d = (Y - T) * M
    q = torch.nn.functional.pad(d * d * float(inv), (0, -n % 32)).reshape(-1, 32)
    while q.shape[1] > 1:
        h = q.shape[1] // 2
        q = q[:, :h] + q[:, h:]
    # FP64 sums of positive terms in another order: 1e-16 a term, far inside 1e-12
    assert abs(float(loss) - float(q.double().sum())) <= 1e-12 * float(loss) + 1e-300


@pytest.mark.parametrize("m,n,k", [(4, 4, 4), (128, 64, 16), (132, 68, 20), (260, 60, 100), (8, 256, 252)])
def test_gemm_of_four_neighbours_equals_the_scalar_one(m, n, k):
    """Packed rows of 4 elements take 16-byte loads; one element of padding or of offset does not."""
    import torch
    from mmd import _native
    from mmd.guess import DensityMLP
    L = _native.lib()
    DensityMLP._sig(L)
    st = _native.stream_ptr()
    g = torch.Generator(device="cuda").manual_seed(m)
    for a16, b16 in ((0, 0), (1, 0), (0, 1)):
        for ta in (0, 1):
            for tb in (0, 1):
                A = torch.randn(*((k, m) if ta else (m, k)), generator=g, device="cuda")
                B = torch.randn(*((n, k) if tb else (k, n)), generator=g, device="cuda")
                A, B = A.bfloat16() if a16 else A, B.bfloat16() if b16 else B
                out = []
                for pad, off in ((0, 0), (1, 0), (0, 1)):
                    args = []
                    for x in (A, B):
                        w = torch.zeros(x.shape[0] * (x.shape[1] + pad) + off, dtype=x.dtype, device="cuda")
                        w[off:].view(x.shape[0], -1)[:, :x.shape[1]] = x
                        args.append((w[off:], x.shape[1] + pad))
                    C = torch.empty(m, n, device="cuda")
                    assert L.mmdg_mlp_gemm(m, n, k, _p(args[0][0]), args[0][1], ta, a16, _p(args[1][0]), args[1][1], tb,
                                           b16, _p(C), n, 0.0, st) == 0
                    out.append(C)
                assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])  # the same sums in the same order

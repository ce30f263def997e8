"""A context's side streams belong to all its callers: one thread captures Fock graphs while
another asks for the ERI tensor and the gradient of the same context."""
import ctypes
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WATER = "\n0 1\nO 0.0 -0.075791844 0.0\nH 0.866811829 0.601435779 0.0\nH -0.866811829 0.601435779 0.0\n"


def _setup():
    import torch
    from mmd import _native
    from mmd.molecule import Molecule
    mol = Molecule(WATER, "6-31g")
    ctx, N = mol.context, mol.nbasis
    A = np.random.default_rng(N).standard_normal((N, N))
    P = torch.as_tensor(0.5 * (A + A.T), device="cuda")
    T = torch.empty(N ** 4, dtype=torch.float64, device="cuda")
    atom = np.array([0, 0, 0, 0, 0, 1, 1, 2, 2], dtype=np.int32)[:ctx.nshell]
    xyz = np.array([a.origin for a in mol.atoms], dtype=np.float64).reshape(-1)
    Z = np.array([8.0, 1.0, 1.0])
    grad = np.zeros(9)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def gradient():
        _native.check(_native.lib().mmdg_rhf_gradient(ctx._h, p(P), p(P), 3, _native._ptr(xyz), _native._ptr(Z),
                                                      _native._ptr(atom), 0.0, _native._ptr(grad),
                                                      _native.stream_ptr()), "mmdg_rhf_gradient")
        return grad.copy()

    def graph(G, tol):
        _native.check(_native.lib().mmdg_fock_graph(ctx._h, p(P), p(G), tol, 0.0, _native.stream_ptr()), "mmdg_fock_graph")

    return ctx, P, T, gradient, graph


def test_fock_capture_beside_tensor_and_gradient():
    import torch
    ctx, P, T, gradient, graph = _setup()
    T0, g0 = ctx.eri_tensor(T).clone(), gradient()
    G0 = ctx.fock(P.reshape(-1), torch.empty_like(P).reshape(-1)).clone()
    torch.cuda.synchronize()
    errors, stop = [], threading.Event()

    def capture():
        try:
            G = torch.empty_like(P)
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in range(1000):  # another threshold: captured anew
                    graph(G, 1e-12 if k % 2 else 1.1e-12)
                graph(G, 1e-12)
                torch.cuda.current_stream().synchronize()
            # G is a sum of up to N^2 ERIs in an order that the atomics choose
            assert float((G.reshape(-1) - G0).abs().max()) < 1e-12
        except Exception as e:  # noqa: BLE001 -- reported by the test's thread
            errors.append(("capture", e))
        finally:
            stop.set()

    def others():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                while not stop.is_set():
                    T.fill_(7.0)
                    for _ in range(20):
                        ctx.eri_tensor(T)
                    torch.cuda.current_stream().synchronize()
                    assert torch.equal(T, T0.reshape(-1))
                    assert np.abs(gradient() - g0).max() < 1e-11
        except Exception as e:  # noqa: BLE001
            errors.append(("others", e))

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        ts = [threading.Thread(target=f) for f in (capture, others)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors


def test_tensor_while_the_caller_has_a_fock_build_in_capture():
    import torch
    ctx, P, T, _, _ = _setup()
    T0 = ctx.eri_tensor(T).clone()
    G = torch.empty_like(P).reshape(-1)
    G0 = ctx.fock(P.reshape(-1), G).clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    cuda_graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cuda_graph, capture_error_mode="thread_local"):
        ctx.fock(P.reshape(-1), G)
        done = []

        def tensor():  # another thread, another stream: not part of the capture
            with torch.cuda.stream(side):
                T.fill_(7.0)
                ctx.eri_tensor(T)
                side.synchronize()
                done.append(torch.equal(T, T0.reshape(-1)))

        t = threading.Thread(target=tensor)
        t.start()
        t.join()
    assert done == [True]
    G.fill_(0.0)
    cuda_graph.replay()
    torch.cuda.synchronize()
    assert float((G - G0).abs().max()) < 1e-12

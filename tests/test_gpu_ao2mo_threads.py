"""Two threads transform tensors of different sizes at the same time: launches of different
shared-memory sizes of one kernel, whose limit is the device's."""
import sys
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_two_threads_with_different_sizes():
    import torch
    from mmd import _native
    sizes, out, errors = (8, 65), {}, []
    data = {}
    for N in sizes:
        g = torch.Generator(device="cuda").manual_seed(N)
        T = torch.randn(N ** 4, generator=g, device="cuda", dtype=torch.float64)
        C = torch.randn(N, N, generator=g, device="cuda", dtype=torch.float64)
        data[N] = (C, T, _native.ao2mo(C, T))
    torch.cuda.synchronize()
    start = threading.Barrier(2)

    def work(N, calls):
        try:
            C, T, _ = data[N]
            buf, tmp = torch.empty_like(T), torch.empty_like(T)
            s = torch.cuda.Stream()
            start.wait()
            with torch.cuda.stream(s):
                for _ in range(calls):
                    _native.ao2mo(C, T, buf, tmp)
            s.synchronize()
            out[N] = buf
        except Exception as e:  # noqa: BLE001 -- reported by the test's thread
            errors.append((N, e))

    ts = [threading.Thread(target=work, args=(N, c)) for N, c in zip(sizes, (8000, 800))]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors
    for N in sizes:
        assert torch.equal(out[N], data[N][2])  # the same integer sums, rounded once

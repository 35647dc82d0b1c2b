"""A caller's streams of every kind: their handles, and what other threads do meanwhile."""
import numpy as np
import pytest

import poissonreconstruction_b200 as prb
from poissonreconstruction_b200 import synthetic

pytestmark = pytest.mark.gpu

LEGACY, PER_THREAD = 1, 2  # cudaStreamLegacy; cudaStreamPerThread: another stream in every host thread


def test_staged_host_copies_on_the_per_thread_stream(ctx):
    """The helper threads of a staged copy (32 MiB and more in, 8 MiB and more out) do not use the
    context's stream handle, which names another stream there: the results are those of a context
    with a stream of its own."""
    pts = synthetic.sphere(700_001, seed=77)
    queries = np.ascontiguousarray(synthetic.sphere(1000, seed=78)[:, :3])
    params = prb.ReconstructParams(depth=7, point_weight=4.0)

    def results(c):
        c.solve(pts, params)
        return (c.coefficients(),) + tuple(c.loss_backward(queries)[:3])

    expected = results(ctx)
    with prb.Context(0, stream=PER_THREAD) as c:
        for _ in range(3):
            for got, want in zip(results(c), expected):
                assert np.array_equal(got, want)


def _blocking_stream():
    """A stream that orders with the legacy default stream (cudaStreamDefault)."""
    import ctypes
    import torch
    torch.zeros(1, device="cuda")
    s = ctypes.c_void_p()
    assert ctypes.CDLL("libcuda.so.1").cuStreamCreate(ctypes.byref(s), 0) == 0
    return s.value


@pytest.mark.parametrize("stream", ["legacy", "per-thread", "blocking"])
@pytest.mark.parametrize("degree,depth", [(1, 3), (1, 6), (2, 5), (2, 6)])
def test_every_kind_of_stream_handle(ctx, degree, depth, stream):
    """A solver's first solve, its first and its later replays give the same bits on each of them."""
    handle = {"legacy": LEGACY, "per-thread": PER_THREAD}.get(stream) or _blocking_stream()
    with prb.Context(0, stream=handle) as c:
        for seed in (5, 6, 5):
            pts = synthetic.torus(3000, seed=seed)
            params = prb.ReconstructParams(depth=depth, degree=degree, point_weight=4.0)
            st, expected = c.solve(pts, params), ctx.solve(pts, params)
            assert st.pcg_iterations == expected.pcg_iterations
            assert np.array_equal(c.coefficients(), ctx.coefficients())


@pytest.mark.parametrize("degree", [1, 2])
def test_capture_beside_a_thread_on_the_legacy_stream(degree):
    """While a stream that orders with the legacy stream is being captured, no thread of the process may
    use the legacy stream: a context on such a stream does not capture it.  (A new point weight is a new
    capture.)"""
    import threading
    import torch
    x = torch.zeros(16, device="cuda")
    stop, failed = threading.Event(), []

    def work():
        try:
            while not stop.is_set():
                x.add_(1.0)
        except Exception as e:
            failed.append(e)

    pts = synthetic.torus(3000, seed=7)
    with prb.Context(0, stream=_blocking_stream()) as c:
        c.solve(pts, prb.ReconstructParams(depth=6, degree=degree, point_weight=1.0))
        t = threading.Thread(target=work)
        t.start()
        try:
            for k in range(30):
                st = c.solve(pts, prb.ReconstructParams(depth=6, degree=degree, point_weight=2.0 + 0.1 * k))
                assert st.converged == 1
        finally:
            stop.set()
            t.join()
    torch.cuda.synchronize()
    assert not failed, failed

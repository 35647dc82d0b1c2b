"""A caller's streams of every kind: their handles, and what other threads do meanwhile."""
import numpy as np
import pytest

import poissonreconstruction_b200 as prb
from poissonreconstruction_b200 import synthetic

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread: another stream in every host thread


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

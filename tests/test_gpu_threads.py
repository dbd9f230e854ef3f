"""One context per host thread: calls of different sizes at the same time, as include/parhde.h allows."""
import threading

import numpy as np
import pytest

from icpp_2020_parhde_gb300 import Context, graphs
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _both(work):
    """Runs work(0) and work(1) on two threads at once and raises what either raised."""
    errors = []
    ready = threading.Barrier(2)

    def body(i):
        try:
            ready.wait()
            work(i)
        except Exception as e:  # handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=body, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_searches_of_two_sizes_on_two_threads():
    """The searches on one cluster take shared memory by the graph's size: neither thread's limit reaches the other's
    launches, and both get the oracle's pivots."""
    gs = [graphs.mesh(400, 300, seed=1), graphs.mesh(12, 9, seed=2)]
    want = [orc.kcenters(g, 2, 0, parallel=True)[1] for g in gs]

    def work(i):
        with Context(0) as ctx:
            ctx.upload(gs[i])
            for _ in range((60, 1500)[i]):
                assert np.array_equal(ctx.kcenters(2, 0, want_dist=False)[1], want[i])

    _both(work)


def test_batches_of_two_sizes_on_two_threads(monkeypatch):
    """One CTA per graph, with the visited bitmap of the batch's largest graph in shared memory."""
    monkeypatch.setenv("PHDE_BATCH_BFS", "blocks")
    batches = [[graphs.mesh(300, 300, seed=3)] * 2, [graphs.mesh(8, 8, seed=4)] * 2]
    want = []
    for b in batches:
        with Context(0) as ctx:
            ctx.upload_batch(b)
            want.append(ctx.layout_batched(4, 2)[0][0].copy())

    def work(i):
        with Context(0) as ctx:
            for _ in range((15, 200)[i]):
                ctx.upload_batch(batches[i])  # the pipeline is launched or captured anew after an upload
                got = ctx.layout_batched(4, 2)[0]
                np.testing.assert_allclose(np.abs(got[0]), np.abs(want[i]), rtol=0, atol=1e-4)

    _both(work)

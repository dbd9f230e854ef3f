"""The ordered FP64 sums of PivotMDS and PHDE (C^T C and the coordinates' norms in the reference's one-thread order):
bit for bit the oracle's, at the chunk edges of the parallel evaluation and where partial sums cross zero."""
import numpy as np
import pytest

from icpp_2020_parhde_gb300 import graphs
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["PivotMDS", "PHDE"])
@pytest.mark.parametrize("make,k", [
    (lambda: graphs.mesh(8, 8, seed=1), 3),        # one short chunk
    (lambda: graphs.mesh(89, 23, seed=2), 4),      # n = 2047, 2048, 2049: around one chunk
    (lambda: graphs.mesh(64, 32, seed=3), 4),
    (lambda: graphs.mesh(683, 3, seed=4), 4),
    (lambda: graphs.mesh(192, 11, seed=5), 5),     # n = 2112: a chunk and the serial steps' length
    (lambda: graphs.rgg(30000, dim=2, avg_degree=8, seed=6), 10),
    (lambda: graphs.rmat(14, seed=7), 33),         # more than one tile of columns
    (lambda: graphs.grid3d(25, weighted=False), 6),
], ids=["n64", "n2047", "n2048", "n2049", "n2112", "rgg2d", "rmat14", "grid25"])
def test_ordered_sums_bitwise(gpu_ctx, algo, make, k):
    g = make()
    gpu_ctx.upload(g)
    r = gpu_ctx.layout(algo, "Kcenters", k=k, c=2, eig="exact", extra=True)
    L = orc.layout(g, algo, "Kcenters", k, 2, eig="exact", nthreads=1)
    assert np.array_equal(r.sources, L.sources)
    assert np.array_equal(r.basis, L.S)
    C = r.basis
    want = np.empty((k, k))
    for p in range(k):
        for q in range(k):
            want[p, q] = np.add.accumulate(C[:, p] * C[:, q])[-1]  # one addition at a time, each rounded
    assert np.array_equal(r.gram, want)
    # the norms: the same accumulation over the coordinates the GPU's own eigenvectors give
    X = np.zeros((g.n, 2))
    for t in range(2):
        y = r.evecs[:, k - 1 - t]
        for j in range(k):
            X[:, t] = X[:, t] + C[:, j] * y[j]
        X[:, t] *= 1.0 / np.sqrt(np.add.accumulate(X[:, t] * X[:, t])[-1])
    assert np.array_equal(r.coords, X)


def comet(n: int, tail: int):
    """A path of `tail` vertices, numbered from its far end, to a hub with the other vertices as leaves: the first terms
    of the sums are the large ones, so that the rest of a sum stays in one binade."""
    lo = np.concatenate([np.arange(tail), np.full(n - tail - 1, tail)])
    hi = np.concatenate([np.arange(1, tail + 1), np.arange(tail + 1, n)])
    return graphs._csr_from_undirected(n, lo, hi)


@pytest.mark.parametrize("algo", ["PivotMDS", "PHDE"])
@pytest.mark.parametrize("n,tail", [(n, 12) for n in (31, 32, 33)] +
                         [(n, 30) for n in (1055, 1056, 1057, 1087, 1088, 1089, 2079, 2080, 2081)])
def test_ordered_sums_at_the_chunks_edges(gpu_ctx, algo, n, tail):
    """A sum starts with 32 terms one by one and goes on in chunks of 1024: sums that end there, one term before and one
    after, and 32 terms later."""
    g = comet(n, tail)
    gpu_ctx.upload(g)
    k = 3
    r = gpu_ctx.layout(algo, "Kcenters", k=k, c=2, eig="exact", extra=True)
    C = r.basis
    assert np.array_equal(C, orc.layout(g, algo, "Kcenters", k, 2, eig="exact", nthreads=1).S)
    want = np.array([[np.add.accumulate(C[:, p] * C[:, q])[-1] for q in range(k)] for p in range(k)])
    assert np.array_equal(r.gram, want)
    X = np.zeros((n, 2))
    for t in range(2):
        y = r.evecs[:, k - 1 - t]
        for j in range(k):
            X[:, t] = X[:, t] + C[:, j] * y[j]
        X[:, t] *= 1.0 / np.sqrt(np.add.accumulate(X[:, t] * X[:, t])[-1])
    assert np.array_equal(r.coords, X)

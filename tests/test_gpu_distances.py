"""GPU distance kernels against the reference's own distance columns (golden fixtures) and the oracle:
bit-exact hop counts and weighted distances, identical Kcenters pivot order."""
import numpy as np
import pytest

from conftest import GOLDEN_NAMES, golden_runs, load_golden
from icpp_2020_parhde_gb300 import DOBFS, DeltaStep, ParHDEError, graphs
from icpp_2020_parhde_gb300.csr_io import CSRGraph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", GOLDEN_NAMES)
def test_distances_bit_exact_vs_reference(gpu_ctx, name):
    g, rec = load_golden(name)
    gpu_ctx.upload(g)
    d = gpu_ctx.distances(rec["bfs_src"])
    assert d.dtype == np.int32
    assert np.array_equal(d, rec["bfs_dist"])


@pytest.mark.parametrize("case", [c for c in golden_runs()], ids=lambda c: "%s-%s-k%d-c%d" % c)
def test_kcenters_pivot_order_vs_reference(gpu_ctx, case):
    name, algo, k, c = case
    g, rec = load_golden(name)
    ref = rec[f"{algo}_k{k}_c{c}_sources"]
    gpu_ctx.upload(g)
    if algo == "wParHDE":
        pytest.skip("WParHDE interleaves selection with orthogonalisation; covered by the layout tests")
    passes = 3 * k if algo == "ParHDE" else k
    D, src = gpu_ctx.kcenters(passes, 0 if algo == "ParHDE" else 2)
    assert np.array_equal(src, ref[:passes])
    Do, so = orc.kcenters(g, passes, 0 if algo == "ParHDE" else 2)
    assert np.array_equal(D, Do)


@pytest.mark.parametrize("make", [
    lambda: graphs.rmat(16, seed=1),
    lambda: graphs.rgg(60000, dim=2, avg_degree=8, seed=2),
    lambda: graphs.rgg(40000, dim=3, avg_degree=12, seed=3),
    lambda: graphs.mesh(300, 200, seed=4),
], ids=["rmat16", "rgg2d", "rgg3d", "mesh300x200"])
def test_bfs_and_kcenters_exact_vs_oracle(gpu_ctx, make):
    g = make()
    gpu_ctx.upload(g)
    rng = np.random.default_rng(5)
    src = rng.integers(0, g.n, size=4)
    d = gpu_ctx.distances(src)
    for i, s in enumerate(src):
        assert np.array_equal(d[:, i], orc.bfs(g, int(s)))
    D, s = gpu_ctx.kcenters(24, 0)
    Do, so = orc.kcenters(g, 24, 0, parallel=True)
    assert np.array_equal(s, so) and np.array_equal(D, Do)


@pytest.mark.parametrize("L,seed", [(20, 1), (32, 2)])
def test_sssp_exact_vs_oracle(gpu_ctx, L, seed):
    g = graphs.grid3d(L, seed=seed)
    gpu_ctx.upload(g)
    src = [0, g.n - 1, g.n // 2]
    d = gpu_ctx.distances(src)
    for i, s in enumerate(src):
        assert np.array_equal(d[:, i], orc.sssp(g, s))


@pytest.mark.parametrize("local,ctas,delta", [("0", "2", None), ("1", "1", None), ("4", "2", "40"), ("16", "1", "7")])
def test_sssp_round_shapes_exact(gpu_ctx, monkeypatch, local, ctas, delta):
    """The block-local round count, resident CTAs per SM and band width change the work, never the
    distances: a weighted grid and a weighted R-MAT (hubs: several chunks per block) under each shape."""
    monkeypatch.setenv("PHDE_SSSP_LOCAL", local)
    monkeypatch.setenv("PHDE_SSSP_CTAS", ctas)
    if delta is None:
        monkeypatch.delenv("PHDE_SSSP_DELTA", raising=False)
    else:
        monkeypatch.setenv("PHDE_SSSP_DELTA", delta)
    for g in (graphs.grid3d(24, seed=4), graphs.with_random_weights(graphs.rmat(13, seed=5), seed=6, wmin=1, wmax=300)):
        gpu_ctx.upload(g)
        src = [0, g.n - 1, g.n // 3]
        d = gpu_ctx.distances(src)
        for i, s in enumerate(src):
            assert np.array_equal(d[:, i], orc.sssp(g, s))


def test_sssp_exact_on_weighted_rmat(gpu_ctx):
    g = graphs.with_random_weights(graphs.rmat(14, seed=9), seed=3, wmin=1, wmax=1000)
    gpu_ctx.upload(g)
    d = gpu_ctx.distances([0, 17, 999])
    for i, s in enumerate([0, 17, 999]):
        assert np.array_equal(d[:, i], orc.sssp(g, s))


def _two_triangles(weighted=False):
    off = np.array([0, 2, 4, 6, 8, 10, 12], dtype=np.uint32)
    adj = np.array([1, 2, 0, 2, 0, 1, 4, 5, 3, 5, 3, 4], dtype=np.uint32)
    w = np.full(12, 3, dtype=np.int32) if weighted else None
    return CSRGraph(off, adj, w)


def test_disconnected_distances_and_layout_error(gpu_ctx):
    g = _two_triangles()
    gpu_ctx.upload(g)
    d = gpu_ctx.distances([0])
    assert list(d[:, 0]) == [0, 1, 1, -1, -1, -1]
    with pytest.raises(ParHDEError) as e:
        gpu_ctx.layout("ParHDE", k=2, c=2)
    assert e.value.status == -3
    gw = _two_triangles(weighted=True)
    gpu_ctx.upload(gw)
    d = gpu_ctx.distances([4])
    assert list(d[:, 0]) == [orc.SSSP_INF] * 3 + [3, 0, 3]


def test_reference_shaped_dobfs_and_deltastep():
    g = _two_triangles()
    dists = np.full(6, -7.0)
    DOBFS(g.offsets, g.adj, 1, 6, 12, dists)
    assert list(dists) == [1, 0, 1, -7, -7, -7]  # unreached entries untouched (bfs.cc:144-185)
    gw, rec = load_golden("grid12w")
    dist = np.zeros(gw.n)
    DeltaStep(gw.offsets, gw.adj, gw.weights, 1000, gw.n, gw.nnz, dist, 10000)
    assert np.array_equal(dist.astype(np.int32), rec["bfs_dist"][:, 1])


def test_csr_validation_rejects_bad_input(gpu_ctx):
    off = np.array([0, 2, 1, 3], dtype=np.uint32)  # decreasing offsets
    adj = np.array([1, 2, 0], dtype=np.uint32)
    with pytest.raises(ParHDEError) as e:
        gpu_ctx.upload(CSRGraph(off, adj))
    assert e.value.status == -2
    off = np.array([0, 1, 2], dtype=np.uint32)
    adj = np.array([1, 5], dtype=np.uint32)  # neighbour out of range
    with pytest.raises(ParHDEError) as e:
        gpu_ctx.upload(CSRGraph(off, adj))
    assert e.value.status == -2


def test_bounded_wait_times_out_and_context_survives(gpu_ctx):
    assert gpu_ctx.selftest_barrier_timeout(50) == -8  # PHDE_ERR_TIMEOUT
    g, rec = load_golden("mesh125")
    gpu_ctx.upload(g)
    assert np.array_equal(gpu_ctx.distances(rec["bfs_src"]), rec["bfs_dist"])


@pytest.mark.parametrize("nsrc", [5, 64, 100, 300])
def test_multi_source_bfs_bit_exact(gpu_ctx, nsrc):
    """phde_distances with several sources runs the bitset multi-source BFS (up to 256 sources per sweep)."""
    g = graphs.rmat(15, seed=12)
    gpu_ctx.upload(g)
    rng = np.random.default_rng(nsrc)
    src = rng.integers(0, g.n, size=nsrc)
    src[1] = src[0]  # a repeated source is allowed
    d = gpu_ctx.distances(src)
    for i in range(0, nsrc, max(1, nsrc // 7)):
        assert np.array_equal(d[:, i], orc.bfs(g, int(src[i]))), i
    assert np.array_equal(d[:, 0], d[:, 1])


@pytest.mark.parametrize("window", ["0", "1"])
@pytest.mark.parametrize("make,nsrc", [
    (lambda: graphs.rgg(40000, dim=3, avg_degree=12, seed=3), 256),
    (lambda: graphs.rgg(30000, dim=2, avg_degree=8, seed=5), 100),
    (lambda: graphs.rmat(14, seed=2), 256),
], ids=["rgg3d-256", "rgg2d-100", "rmat14-256"])
def test_multi_source_bfs_window_modes(gpu_ctx, monkeypatch, make, nsrc, window):
    """Dense levels with and without the shared-memory frontier window (chosen by index locality; forced here
    both ways, also on the R-MAT graph whose numbering is not local) give the one-source BFS columns."""
    monkeypatch.setenv("PHDE_MSBFS_WINDOW", window)
    g = make()
    gpu_ctx.upload(g)
    rng = np.random.default_rng(nsrc + 7)
    src = rng.integers(0, g.n, size=nsrc)
    d = gpu_ctx.distances(src)
    for i in range(0, nsrc, max(1, nsrc // 9)):
        assert np.array_equal(d[:, i], orc.bfs(g, int(src[i]))), i


def test_multi_source_bfs_on_mesh_and_disconnected(gpu_ctx):
    g, rec = load_golden("mesh125")
    gpu_ctx.upload(g)
    src = np.concatenate([rec["bfs_src"], np.arange(0, 15625, 1000)])
    d = gpu_ctx.distances(src)
    assert np.array_equal(d[:, :3], rec["bfs_dist"])
    for i in range(3, len(src)):
        assert np.array_equal(d[:, i], orc.bfs(g, int(src[i])))
    g2 = _two_triangles()
    gpu_ctx.upload(g2)
    d = gpu_ctx.distances([0, 1, 3, 5])
    assert list(d[:, 0]) == [0, 1, 1, -1, -1, -1] and list(d[:, 2]) == [-1, -1, -1, 0, 1, 1]


def _tree_of_levels(edges, n):
    e = np.asarray(edges, dtype=np.int64)
    return graphs._csr_from_undirected(n, e.min(axis=1), e.max(axis=1))


def _two_stars(leaves: int, tail: int):
    """Stars around A = 0 and B = 1, both joined to m = 2, which carries a path of `tail` vertices.  From a leaf the
    stars' leaves are two levels apart; from the path's end they are one level of 2 * leaves vertices."""
    e = [(0, 2), (1, 2)]
    e += [(2 if i == 0 else 2 + i, 3 + i) for i in range(tail)]
    first = 3 + tail
    e += [(0, first + i) for i in range(leaves)] + [(1, first + leaves + i) for i in range(leaves)]
    return _tree_of_levels(e, first + 2 * leaves)


@pytest.mark.parametrize("make", [
    lambda: graphs.path_graph(33),
    lambda: graphs.mesh(37, 15, seed=7),                        # 17 words: most CTAs of the cluster own one
    lambda: graphs.mesh(512, 3, seed=8),
    lambda: _two_stars(511, 20),                                # rows at the whole-CTA threshold and past it
    lambda: _two_stars(700, 20),
    lambda: _two_stars(2048, 20),                               # 4096 vertices in one level: the cluster's limit
    lambda: _two_stars(3000, 20),                               # past it in the second pass: the grid goes on
    lambda: graphs.mesh(1000, 900, seed=9),                     # row starts no longer in shared memory
], ids=["path33", "mesh37x15", "mesh512x3", "stars511", "stars700", "stars2048", "stars3000", "mesh1000x900"])
@pytest.mark.parametrize("variant", [0, 2])
def test_cluster_kcenters_exact_vs_oracle(gpu_ctx, make, variant):
    """The searches on one thread-block cluster, and their continuation by the whole grid after a wide level: the
    oracle's pivots and distances."""
    g = make()
    gpu_ctx.upload(g)
    passes = 12
    D, s = gpu_ctx.kcenters(passes, variant)
    Do, so = orc.kcenters(g, passes, variant, parallel=True)
    assert np.array_equal(s, so) and np.array_equal(D, Do)


def test_cluster_kcenters_duplicate_sources_and_fixed_sources(gpu_ctx):
    """More passes than vertices (the duplicate fix-up) and fixed sources, a vertex out of reach among them."""
    g = graphs.path_graph(9)
    gpu_ctx.upload(g)
    D, s = gpu_ctx.kcenters(12, 0)
    Do, so = orc.kcenters(g, 12, 0)
    assert np.array_equal(s, so) and np.array_equal(D, Do)
    two = _tree_of_levels([(i, i + 1) for i in range(60)] + [(61 + i, 62 + i) for i in range(10)], 72)
    gpu_ctx.upload(two)
    d = gpu_ctx.distances([5, 65])
    assert np.array_equal(d[:, 0], orc.bfs(two, 5)) and np.array_equal(d[:, 1], orc.bfs(two, 65))
    with pytest.raises(ParHDEError):
        gpu_ctx.kcenters(3, 0)


@pytest.mark.parametrize("make", [
    lambda: graphs.path_graph(700),
    lambda: graphs.mesh(60, 41, seed=21),                             # at most 8 neighbours: eight lanes
    lambda: graphs.rgg(9000, dim=2, avg_degree=5, seed=22),           # up to 16: sixteen lanes
    lambda: graphs.rgg(20000, dim=2, avg_degree=9, seed=23),          # up to 32: two edges per lane
    lambda: _two_stars(31, 5),                                        # rows of exactly 32
    lambda: _two_stars(32, 5),                                        # 33: the edge-balanced kernel
], ids=["path700", "mesh60x41", "rgg5", "rgg9", "deg32", "deg33"])
@pytest.mark.parametrize("ctas,delta", [("1", None), ("2", "100")])
def test_sssp_lane_groups_exact(gpu_ctx, monkeypatch, make, ctas, delta):
    """The lane-group kernel in each of its shapes, with the wide band and with many bands."""
    monkeypatch.setenv("PHDE_SSSP_CTAS", ctas)
    if delta:
        monkeypatch.setenv("PHDE_SSSP_DELTA", delta)
    else:
        monkeypatch.delenv("PHDE_SSSP_DELTA", raising=False)
    g = graphs.with_random_weights(make(), seed=3)
    gpu_ctx.upload(g)
    src = [0, g.n // 3, g.n - 1]
    d = gpu_ctx.distances(src)
    for i, s in enumerate(src):
        assert np.array_equal(d[:, i], orc.sssp(g, s))


@pytest.mark.parametrize("make", [
    lambda width: graphs.star_graph(width),
    lambda width: graphs.star_graph(width + 1),
    lambda width: graphs.rmat(18, seed=4),  # above 24 neighbours a vertex: every level on the whole grid
], ids=["grid-wide-star", "one-more", "rmat18"])
def test_kcenters_levels_of_one_and_more_grid_iterations(gpu_ctx, make):
    """Levels that fit one iteration of the grid push their vertices at once, wider ones list them first: stars
    whose one level takes exactly the grid's threads and one more, and an R-MAT with levels of both kinds."""
    import torch
    g = make(torch.cuda.get_device_properties(0).multi_processor_count * 1024)
    gpu_ctx.upload(g)
    D, s = gpu_ctx.kcenters(4, 0)
    Do, so = orc.kcenters(g, 4, 0, parallel=True)
    assert np.array_equal(s, so) and np.array_equal(D, Do)


def _hub_mesh(nx: int, ny: int, leaves: int):
    """A mesh whose last vertex carries `leaves` leaves: narrow levels, then one wide one."""
    g = graphs.mesh(nx, ny, seed=31)
    src = np.repeat(np.arange(g.n), np.diff(g.offsets.astype(np.int64)))
    keep = src < g.adj
    lo = np.concatenate([src[keep], np.full(leaves, g.n - 1)])
    hi = np.concatenate([g.adj[keep].astype(np.int64), g.n + np.arange(leaves)])
    return graphs._csr_from_undirected(g.n + leaves, lo, hi)


@pytest.mark.parametrize("nx,ny,leaves", [(100, 100, 5000), (37, 20, 4097), (500, 400, 30000), (100, 100, 250_000)])
def test_wide_level_continues_on_the_grid(gpu_ctx, nx, ny, leaves):
    """A level too wide for the cluster goes on from there on the whole grid: the oracle's distances, from sources
    before, at and behind the wide level, and the levels before it are not searched again."""
    g = _hub_mesh(nx, ny, leaves)
    gpu_ctx.upload(g)
    for s in (0, nx * ny - 1, g.n - 1):
        assert np.array_equal(gpu_ctx.distances([s])[:, 0], orc.bfs(g, s))
    D, src = gpu_ctx.kcenters(5, 0)
    Do, so = orc.kcenters(g, 5, 0, parallel=True)
    assert np.array_equal(src, so) and np.array_equal(D, Do)
    if leaves * 6 < g.nnz:  # the hub's level is no bottom-up step
        # the first pass crosses the mesh before the hub: begun again, it would add the mesh's entries (over 0.8 nnz).
        # A bottom-up level may read a row that the next reads again, at most in the last levels: half a pass is left.
        r = gpu_ctx.layout("ParHDE", "Kcenters", k=2, c=2)
        assert 0 < r.stats["edges_examined"] <= 6.5 * g.nnz


@pytest.mark.parametrize("ny", [1536, 1537], ids=["3<<20", "past it"])
def test_cluster_size_limit(gpu_ctx, ny):
    """Meshes of the most vertices the cluster takes and of more, which stay on the grid."""
    g = graphs.mesh(2048, ny, seed=33)
    gpu_ctx.upload(g)
    before = gpu_ctx.launch_count
    D, s = gpu_ctx.kcenters(2, 0)
    launches = gpu_ctx.launch_count - before
    Do, so = orc.kcenters(g, 2, 0, parallel=True)
    assert np.array_equal(s, so) and np.array_equal(D, Do)
    before = gpu_ctx.launch_count
    gpu_ctx.kcenters(2, 0)
    assert gpu_ctx.launch_count - before == launches == (3 if g.n == 3 << 20 else 2)  # fill, (cluster), grid


@pytest.mark.parametrize("make", [lambda: graphs.rmat(11, seed=5), lambda: graphs.mesh(30, 20, seed=6)],
                         ids=["edge-balanced", "lane-groups"])
def test_sssp_first_search_on_a_graph_launches_no_more_than_the_next(gpu_ctx, make):
    """The kernel is picked by what the upload found: no pass over the graph and no wait before a graph's first search
    (below 2^20 vertices, where the band does not depend on the weights)."""
    g = graphs.with_random_weights(make(), seed=3)
    gpu_ctx.upload(g)
    counts = []
    for _ in range(2):
        before = gpu_ctx.launch_count
        assert np.array_equal(gpu_ctx.distances([1])[:, 0], orc.sssp(g, 1))
        counts.append(gpu_ctx.launch_count - before)
    assert counts[0] == counts[1]


@pytest.mark.parametrize("hub", [32, 33])
def test_sssp_on_a_converted_graph(gpu_ctx, hub):
    """The largest degree is known for graphs made from matrix entries as well."""
    g = graphs.with_random_weights(_two_stars(hub - 1, 5), seed=4)
    src = np.repeat(np.arange(g.n), np.diff(g.offsets.astype(np.int64)))
    low = src > g.adj
    gpu_ctx.graph_from_entries(src[low] + 1, g.adj[low] + 1, g.weights[low], g.n, g.n, True)
    assert np.array_equal(gpu_ctx.distances([3])[:, 0], orc.sssp(g, 3))


@pytest.mark.parametrize("window", ["0", "1"])
@pytest.mark.parametrize("nsrc", [65, 128, 129, 180, 192, 193, 400])
def test_multi_source_bfs_words(gpu_ctx, monkeypatch, nsrc, window):
    """Sweeps at the edges of the frontier words' counts, a second sweep among them: every column against one source."""
    monkeypatch.setenv("PHDE_MSBFS_WINDOW", window)
    g = graphs.rgg(6000, dim=3, avg_degree=10, seed=35)
    gpu_ctx.upload(g)
    src = np.random.default_rng(nsrc).integers(0, g.n, size=nsrc)
    d = gpu_ctx.distances(src)
    for i in range(nsrc):
        assert np.array_equal(d[:, i], orc.bfs(g, int(src[i]))), i


@pytest.mark.parametrize("leaves", [802_000, 818_000, 820_000])
def test_kcenters_bitmaps_around_the_shared_memory_limit(gpu_ctx, leaves):
    """Bottom-up levels whose frontier bitmap just fits the block's shared memory beside the list, and does not."""
    g = graphs.star_graph(leaves)
    gpu_ctx.upload(g)
    D, s = gpu_ctx.kcenters(3, 0)
    Do, so = orc.kcenters(g, 3, 0, parallel=True)
    assert np.array_equal(s, so) and np.array_equal(D, Do)


@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("passes", [4096, 4097, 56_000])
def test_kcenters_with_a_long_history(gpu_ctx, passes, variant):
    """Passes at and past those whose history is in shared memory, and more than shared memory holds."""
    g = graphs.path_graph(9)
    gpu_ctx.upload(g)
    _, s = gpu_ctx.kcenters(passes, variant, want_dist=False)
    assert np.array_equal(s, orc.kcenters(g, passes, variant)[1])


def test_cluster_search_reaches_empty_rows_at_the_end(gpu_ctx):
    """A directed CSR whose last vertices have no neighbours: their rows start past an adjacency of whole pages."""
    spine, width = 512, 1024
    nnz = spine * width  # 2 MiB of adjacency
    nxt = np.arange(1, spine)
    rows, first = [], spine
    for i in range(spine):
        leaves = width if i == spine - 1 else width - 1
        rows.append(np.concatenate([nxt[i: i + 1], np.arange(first, first + leaves)]))
        first += leaves
    off = np.concatenate([np.arange(spine + 1) * width, np.full(first - spine, nnz)])
    g = CSRGraph(off.astype(np.uint32), np.concatenate(rows).astype(np.uint32))
    gpu_ctx.upload(g)
    d = gpu_ctx.distances([0])[:, 0]
    want = np.concatenate([np.arange(spine)] + [np.full(len(r) - (i < spine - 1), i + 1) for i, r in enumerate(rows)])
    assert np.array_equal(d, want)


@pytest.mark.parametrize("more", [-1, 0, 1, 155])
def test_top_down_levels_around_one_grid_iteration(gpu_ctx, monkeypatch, tmp_path, more):
    """Top-down levels with as many out-edges as the grid has threads, one fewer and more: pushed at once, or listed
    first.  A hub with that many neighbours and then its leaves, before a mesh large enough to keep both levels
    top-down; the traced search stays on the grid and says so."""
    import torch
    width = torch.cuda.get_device_properties(0).multi_processor_count * 1024 + more
    body = graphs.mesh(700, 700, seed=36)
    src = np.repeat(np.arange(body.n), np.diff(body.offsets.astype(np.int64)))
    keep = src < body.adj
    first = width + 1  # vertices: the source, the hub, width - 1 leaves, the mesh behind the last leaf
    lo = np.concatenate([[0], np.full(width - 1, 1), [width], src[keep] + first])
    hi = np.concatenate([[1], np.arange(2, width + 1), [first], body.adj[keep].astype(np.int64) + first])
    g = graphs._csr_from_undirected(first + body.n, lo, hi)
    trace = tmp_path / "levels.csv"
    monkeypatch.setenv("PHDE_BFS_TRACE", str(trace))
    gpu_ctx.upload(g)
    D, _ = gpu_ctx.kcenters(1, 0)
    assert np.array_equal(D[:, 0], orc.bfs(g, 0))
    level = [[int(x) for x in line.split(",")] for line in trace.read_text().splitlines()[1:4]]
    assert [(r[3], r[4]) for r in level] == [(0, 0), (1, 0), (2, 0)]  # none of the three is bottom-up
    assert (level[0][5], level[0][6]) == (1, width) and (level[1][5], level[1][6]) == (width - 1, width)

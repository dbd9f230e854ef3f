"""The work this framework is used for, as measurable cases.

``listed()`` names the cases and ``draw(rng)`` gives one more of the same ranges; ``prepare`` makes what a program
has in hand (a synthetic graph generated on the GPU from the seed, uploaded into a Context), ``run`` makes the
public calls and returns their results, ``work`` is what one pass cannot do without, and ``exact`` is the same
result in 64 bits from plain torch on graphs small enough for it.

Graphs are those of the package's own configurations: triangulated meshes, R-MAT (edgefactor 16, .57/.19/.19),
random geometric graphs in 2-D and 3-D, weighted 6-neighbour grids; symmetrised, connected, without loops or
duplicates, vertices numbered as the package's generators number them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from icpp_2020_parhde_gb300 import Context, CSRGraph

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # embed's default options (ParHDE, Kcenters, k = 10, FP64, power iteration) on the 125 x 125 mesh: the
        # smallest everyday call, many short breadth-first levels
        {"name": "mesh125_plain", "kind": "layout", "graph": "mesh", "nx": 125, "ny": 125, "algo": "ParHDE",
         "strategy": "Kcenters", "k": 10, "c": 2, "precision": "fp64", "eig": "power"},
        # the reference's pipeline as it stands on a mid-sized scale-free graph
        {"name": "rmat20_plain", "kind": "layout", "graph": "rmat", "scale": 20, "algo": "ParHDE",
         "strategy": "Kcenters", "k": 50, "c": 3, "precision": "fp64", "eig": "power"},
        # the benchmark's headline: a new graph in pinned host memory, learned pivots, exact-Gram stages, Jacobi
        {"name": "rmat22_learned_upload", "kind": "layout", "graph": "rmat", "scale": 22, "algo": "ParHDE",
         "strategy": "Learned", "k": 64, "c": 3, "precision": "exact", "eig": "exact", "upload": True},
        # the same options on the large high-diameter graph of the learned configuration
        {"name": "rgg3d_8m_learned", "kind": "layout", "graph": "rgg3d", "n": 8_000_000, "algo": "ParHDE",
         "strategy": "Learned", "k": 64, "c": 3, "precision": "exact", "eig": "exact"},
        # a 2-D geometric graph with the mixed-precision pipeline: FP32 stages, high diameter, ragged size
        {"name": "rgg2d_150k_mixed", "kind": "layout", "graph": "rgg2d", "n": 150_001, "algo": "ParHDE",
         "strategy": "Kcenters", "k": 20, "c": 2, "precision": "mixed", "eig": "exact"},
        # WParHDE at its benchmark size: delta-stepping, coupled Gram-Schmidt, weighted Laplacian
        {"name": "grid256_weighted", "kind": "layout", "graph": "grid", "nx": 256, "ny": 256, "nz": 256,
         "algo": "wParHDE", "strategy": "Kcenters", "k": 20, "c": 2, "precision": "fp64", "eig": "power"},
        # WParHDE on an everyday weighted grid with ragged sides
        {"name": "grid65_weighted", "kind": "layout", "graph": "grid", "nx": 65, "ny": 61, "nz": 70,
         "algo": "wParHDE", "strategy": "Kcenters", "k": 20, "c": 2, "precision": "fp64", "eig": "power"},
        # PivotMDS, the reference's other algorithm family (PHDE shares its kernels)
        {"name": "rgg2d_60k_pivotmds", "kind": "layout", "graph": "rgg2d", "n": 60_000, "algo": "PivotMDS",
         "strategy": "Kcenters", "k": 10, "c": 2, "precision": "fp64", "eig": "power"},
        # a collection of graphs laid out by one call: the batched configuration
        {"name": "batch512", "kind": "batch", "count": 512, "nmin": 1000, "nmax": 200_000, "strategy": "Kcenters",
         "k": 10, "c": 2},
        # a smaller collection with learned pivots
        {"name": "batch96_learned", "kind": "batch", "count": 96, "nmin": 1000, "nmax": 50_000,
         "strategy": "Learned", "k": 10, "c": 2},
        # distance columns alone: hop counts from 64 sources
        {"name": "distances_rmat18", "kind": "distances", "graph": "rmat", "scale": 18, "nsrc": 64},
        # the draw tool's image of a scale-free graph
        {"name": "draw_rmat18", "kind": "draw", "graph": "rmat", "scale": 18},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["plain", "exact", "mixed", "learned", "weighted", "mds", "batch", "distances", "draw"])
    k = _log_int(rng, 6, 24)
    c = rng.choice([2, 3])
    if what == "batch":
        return {"kind": "batch", "count": _log_int(rng, 8, 400), "nmin": _log_int(rng, 600, 2000),
                "nmax": _log_int(rng, 4000, 120_000), "strategy": rng.choice(["Kcenters", "Kcenters", "Learned"]),
                "k": _log_int(rng, 6, 16), "c": c}
    if what == "weighted":
        nx, ny, nz = (_log_int(rng, 8, 180) for _ in range(3))
        return {"kind": "layout", "graph": "grid", "nx": nx, "ny": ny, "nz": nz, "algo": "wParHDE",
                "strategy": "Kcenters", "k": k, "c": c, "precision": "fp64", "eig": rng.choice(["power", "exact"])}
    if what == "distances":
        g = rng.choice([{"graph": "rmat", "scale": rng.randint(13, 19)}, {"graph": "rgg2d", "n": _log_int(rng, 1500, 90_000)}])
        return {"kind": "distances", **g, "nsrc": _log_int(rng, 1, 300)}
    if what == "draw":
        g = rng.choice([{"graph": "rmat", "scale": rng.randint(13, 19)}, {"graph": "rgg2d", "n": _log_int(rng, 1500, 900_000)}])
        return {"kind": "draw", **g}
    if what == "mds":
        return {"kind": "layout", "graph": "rgg2d", "n": _log_int(rng, 1500, 120_000),
                "algo": rng.choice(["PivotMDS", "PHDE"]), "strategy": "Kcenters", "k": _log_int(rng, 4, 12), "c": 2,
                "precision": "fp64", "eig": rng.choice(["power", "exact"])}
    o = {"algo": "ParHDE", "c": c}
    if what == "learned":
        g = rng.choice([{"graph": "rmat", "scale": rng.randint(15, 21)}, {"graph": "rgg3d", "n": _log_int(rng, 30_000, 3_000_000)},
                        {"graph": "rgg2d", "n": _log_int(rng, 3000, 150_000)}])
        return {"kind": "layout", **g, **o, "strategy": "Learned", "k": _log_int(rng, 10, 64),
                "precision": rng.choice(["exact", "exact", "mixed"]), "eig": "exact",
                "upload": rng.choice([False, True])}
    g = rng.choice([{"graph": "rmat", "scale": rng.randint(13, 20)}, {"graph": "rgg2d", "n": _log_int(rng, 1500, 200_000)},
                    {"graph": "rgg3d", "n": _log_int(rng, 3000, 700_000)},
                    {"graph": "mesh", "nx": _log_int(rng, 20, 400), "ny": _log_int(rng, 20, 400)}])
    precision, eig = {"plain": ("fp64", "power"), "exact": ("exact", "exact"), "mixed": ("mixed", "exact")}[what]
    return {"kind": "layout", **g, **o, "strategy": rng.choice(["Kcenters", "Kcenters", "RandFine"]), "k": k,
            "precision": precision, "eig": eig}


# ------------------------------------------------------------------------------------------------
# Graphs: (offsets int64 [n + 1], adjacency int64 [nnz], weights int32 [nnz] or None) on the device.

def _gen(seed, salt):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _csr(n, u, v, w=None):
    """Sorted symmetric CSR of the undirected edges {u, v}, loops and duplicates dropped."""
    keep = u != v
    key = (torch.minimum(u, v) * n + torch.maximum(u, v))[keep]
    if w is None:
        key = torch.unique(key)
    else:  # the callers with weights have no duplicates
        key, at = torch.sort(key)
        w = w[keep][at]
    lo, hi = key // n, key % n
    key, at = torch.sort(torch.cat([lo * n + hi, hi * n + lo]))
    off = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
    off[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return off, key % n, None if w is None else torch.cat([w, w])[at]


def _rows(off):
    return torch.repeat_interleave(torch.arange(off.numel() - 1, device=off.device), off[1:] - off[:-1])


def _components(off, adj):
    """The smallest vertex of every vertex's component."""
    n = off.numel() - 1
    src = _rows(off)
    f = torch.arange(n, device=off.device)
    while True:
        gf = f[f]
        least = gf.scatter_reduce(0, src, gf[adj], "amin")
        nf = f.scatter_reduce(0, f, least, "amin")
        nf = torch.minimum(torch.minimum(nf, least), gf)
        if torch.equal(nf, f):
            return f
        f = nf


def _largest(off, adj, n_want):
    """The largest component relabelled in increasing order, brought to n_want vertices: the last leaves go, or new
    leaves hang at the first vertices (a graph has the same number of vertices whatever its seed)."""
    n = off.numel() - 1
    lab = _components(off, adj)
    size = torch.bincount(lab, minlength=n)
    keep = lab == torch.argmax(size)
    over = int(keep.sum()) - n_want
    if over > 0:
        leaves = (keep & (off[1:] - off[:-1] == 1)).nonzero()[:, 0]
        keep[leaves[leaves.numel() - over:]] = False
    new = torch.cumsum(keep, 0) - 1
    src = _rows(off)
    ekeep = keep[src] & keep[adj] & (src < adj)
    u, v = new[src[ekeep]], new[adj[ekeep]]
    if over < 0:
        extra = torch.arange(-over, device=off.device)
        u, v = torch.cat([u, extra]), torch.cat([v, n_want + over + extra])
    return _csr(n_want, u, v)


def _mesh(nx, ny, seed):
    vid = torch.arange(nx * ny, device=DEVICE).reshape(ny, nx)
    coin = torch.rand((ny - 1, nx - 1), generator=_gen(seed, 1), device=DEVICE) < 0.5
    u = [vid[:, :-1].ravel(), vid[:-1].ravel(), torch.where(coin, vid[:-1, :-1], vid[:-1, 1:]).ravel()]
    v = [vid[:, 1:].ravel(), vid[1:].ravel(), torch.where(coin, vid[1:, 1:], vid[1:, :-1]).ravel()]
    return _csr(nx * ny, torch.cat(u), torch.cat(v))


def _rmat(scale, seed):
    g, N = _gen(seed, 2), 1 << scale
    u = torch.zeros(16 * N, dtype=torch.int64, device=DEVICE)
    v = torch.zeros_like(u)
    for level in range(scale):
        r = torch.rand(16 * N, generator=g, device=DEVICE)
        u |= (r >= 0.76).long() << level
        v |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << level
    perm = torch.argsort(torch.rand(N, generator=g, device=DEVICE, dtype=torch.float64))
    off, adj, _ = _csr(N, perm[u], perm[v])
    return _largest(off, adj, _size({"kind": "layout", "graph": "rmat", "scale": scale})[0])


def _grid(nx, ny, nz, seed):
    g = _gen(seed, 3)
    vid = torch.arange(nx * ny * nz, device=DEVICE).reshape(nz, ny, nx)
    u = torch.cat([vid[:-1].ravel(), vid[:, :-1].ravel(), vid[:, :, :-1].ravel()])
    v = torch.cat([vid[1:].ravel(), vid[:, 1:].ravel(), vid[:, :, 1:].ravel()])
    w = torch.randint(1, 256, (u.numel(),), generator=g, device=DEVICE, dtype=torch.int32)
    return _csr(nx * ny * nz, u, v, w)


def _rgg(sizes, dim, degree, seed):
    """Random geometric graphs of the given sizes side by side, each vertex range numbered cell by cell and
    connected by an edge to a vertex close by for every smaller component: (off, adj, None, positions, first
    vertex of every graph)."""
    gen = _gen(seed, 4)
    sizes = torch.tensor(sizes, device=DEVICE)
    n, B = int(sizes.sum()), sizes.numel()
    ball = math.pi if dim == 2 else 4.0 * math.pi / 3.0
    r = (degree / (ball * sizes.double())) ** (1.0 / dim)
    nc = torch.clamp((1.0 / r).long(), min=1)
    first_cell = torch.zeros(B + 1, dtype=torch.int64, device=DEVICE)
    first_cell[1:] = torch.cumsum(nc ** dim, 0)
    gid = torch.repeat_interleave(torch.arange(B, device=DEVICE), sizes)
    pts = torch.rand((n, dim), generator=gen, device=DEVICE, dtype=torch.float64)
    cell = torch.minimum((pts * nc[gid, None]).long(), nc[gid, None] - 1)

    def index(cc, g):
        key = cc[:, 0]
        for d in range(1, dim):
            key = key * nc[g] + cc[:, d]
        return first_cell[g] + key

    at = torch.argsort(pts[:, 0])
    at = at[torch.sort(index(cell, gid)[at], stable=True)[1]]
    pts, cell = pts[at], cell[at]
    begin = torch.zeros(int(first_cell[-1]) + 1, dtype=torch.int64, device=DEVICE)
    begin[1:] = torch.cumsum(torch.bincount(index(cell, gid), minlength=begin.numel() - 1), 0)
    us, vs = [], []
    steps = [(0,), (1,)] if dim == 2 else [(0, 0), (0, 1), (1, -1), (1, 0), (1, 1)]
    for s0 in range(0, n, 1 << 20):
        i = torch.arange(s0, min(n, s0 + (1 << 20)), device=DEVICE)
        for step in steps:  # half of the cells around; the last coordinate's three cells are one range
            lead = cell[i][:, :-1] + torch.tensor(step, device=DEVICE)
            ok = ((lead >= 0) & (lead < nc[gid[i], None])).all(1)
            p, lead = i[ok], lead[ok]
            g, z = gid[p], cell[p][:, -1]
            a = begin[index(torch.cat([lead, torch.clamp(z - 1, min=0)[:, None]], 1), g)]
            b = begin[index(torch.cat([lead, torch.minimum(z + 1, nc[g] - 1)[:, None]], 1), g) + 1]
            if not any(step):
                a = torch.maximum(a, p + 1)  # within the own row of cells every pair once
            cnt = torch.clamp(b - a, min=0)
            who = torch.repeat_interleave(torch.arange(p.numel(), device=DEVICE), cnt)
            j = torch.arange(who.numel(), device=DEVICE) - (torch.cumsum(cnt, 0) - cnt)[who] + a[who]
            u = p[who]
            near = ((pts[u] - pts[j]) ** 2).sum(1) <= (r * r)[gid[u]]
            us.append(u[near])
            vs.append(j[near])
    u, v = torch.cat(us), torch.cat(vs)
    first = torch.zeros(B + 1, dtype=torch.int64, device=DEVICE)
    first[1:] = torch.cumsum(sizes, 0)
    off, adj, _ = _csr(n, u, v)
    root = (_components(off, adj) == torch.arange(n, device=DEVICE)).nonzero()[:, 0]
    root = root[root != first[gid[root]]]  # every other component hangs at the vertex before its first one
    off, adj, _ = _csr(n, torch.cat([u, root]), torch.cat([v, root - 1]))
    return off, adj, None, pts, first


def _graph(case, seed):
    kind = case["graph"]
    if kind == "mesh":
        return _mesh(case["nx"], case["ny"], seed)
    if kind == "rmat":
        return _rmat(case["scale"], seed)
    if kind == "grid":
        return _grid(case["nx"], case["ny"], case["nz"], seed)
    return _rgg([case["n"]], 2 if kind == "rgg2d" else 3, 8.0 if kind == "rgg2d" else 12.0, seed)


def _batch_sizes(case):
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [int(math.exp(x)) for x in np.random.default_rng(1).uniform(lo, hi, case["count"])]


# ------------------------------------------------------------------------------------------------

def _pinned(count, dtype):
    return torch.empty(count, dtype=dtype, pin_memory=torch.cuda.is_available()).numpy()


def _host(t, dtype, pinned=False):
    t = t.to(torch.int32)
    if pinned:
        a = _pinned(t.numel(), torch.int32)
        torch.from_numpy(a).copy_(t)
    else:
        a = t.cpu().numpy()
    return a.view(dtype)


def _host_graph(off, adj, w, pinned=False):
    return CSRGraph(_host(off, np.uint32, pinned), _host(adj, np.uint32, pinned), None if w is None else _host(w, np.int32, pinned))


def prepare(case, seed):
    s = {"case": case, "ctx": Context(0)}
    if case["kind"] == "batch":
        off, adj, _, _, first = _rgg(_batch_sizes(case), 2, 8.0, seed)
        whole, first = _host_graph(off, adj, None), first.tolist()
        graphs = []
        for a, b in zip(first[:-1], first[1:]):
            e0, e1 = int(whole.offsets[a]), int(whole.offsets[b])
            graphs.append(CSRGraph(whole.offsets[a: b + 1] - np.uint32(e0), whole.adj[e0:e1] - np.uint32(a)))
        s["ctx"].upload_batch(graphs)
        s["coords"] = _pinned(first[-1] * case["c"], torch.float64)
    else:
        made = _graph(case, seed)
        g = _host_graph(*made[:3], pinned=bool(case.get("upload")))
        if case.get("upload"):
            s["graph"] = g
        else:
            s["ctx"].upload(g)
        if case["kind"] == "layout":
            s["coords"] = _pinned(g.n * case["c"], torch.float64)
        elif case["kind"] == "distances":
            s["sources"] = np.random.default_rng(seed).integers(0, g.n, case["nsrc"])
        else:  # positions to draw: a geometric graph's own, else hubs near the middle as a spectral layout has them
            if len(made) > 3:
                xy = made[3]
            else:
                deg = (made[0][1:] - made[0][:-1]).double()
                xy = torch.randn((g.n, 2), generator=_gen(seed, 5), device=DEVICE, dtype=torch.float64) / deg.sqrt()[:, None]
            xy = (xy - xy.amin(0)) / (xy.amax(0) - xy.amin(0)) - 0.5  # one aspect, whatever the seed
            xy = xy.cpu().numpy()
            s["x"], s["y"] = np.ascontiguousarray(xy[:, 0]), np.ascontiguousarray(xy[:, 1])
            s["ctx"].draw(s["x"], s["y"])  # the image's size, for the host buffer that it goes to
            W, H = s["ctx"].draw_size
            s["image"] = _pinned(W * H * 4, torch.uint8).reshape(H, W, 4)
    if torch.cuda.is_available():
        torch.cuda.empty_cache()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    if case["kind"] == "batch":
        ctx.layout_batched(k=case["k"], c=case["c"], coords_out=s["coords"], strategy=case["strategy"])
        return {"coords": s["coords"]}
    if case["kind"] == "distances":
        return {"distances": ctx.distances(s["sources"])}
    if case["kind"] == "draw":
        ctx.draw(s["x"], s["y"])
        return {"image": ctx.draw_image(s["image"])}
    if case.get("upload"):
        ctx.upload(s["graph"])
    r = ctx.layout(case["algo"], case["strategy"], k=case["k"], c=case["c"], precision=case["precision"], eig=case["eig"],
                   coords_out=s["coords"])
    return {"coords": r.coords, "sources": r.sources}


# ------------------------------------------------------------------------------------------------

def _size(case):
    """(vertices, about the stored entries) of a case's graph."""
    if case["kind"] == "batch":
        n = sum(_batch_sizes(case))
        return n, 7.95 * n
    kind = case["graph"]
    if kind == "mesh":
        return case["nx"] * case["ny"], 6.0 * case["nx"] * case["ny"]
    if kind == "rmat":
        s = case["scale"]
        return int((0.616 - 0.024 * (s - 20)) * 2.0 ** s), (0.936 + 0.016 * min(s - 20, 3)) * 2.0 ** (s + 5)
    if kind == "grid":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, 6.0 * n
    return case["n"], (7.95 if kind == "rgg2d" else 11.9) * case["n"]


def work(case):
    """The graph read once and the results written once; the products of the basis (Gram-Schmidt against what is
    accepted, L S over the entries, S^T L S, S Y) as operations."""
    n, nnz = _size(case)
    graph = 4 * (n + 1) + 4 * nnz * (2 if case.get("graph") == "grid" else 1)
    if case["kind"] == "distances":
        return {"bytes": graph + 4 * n * case["nsrc"], "flops": 0}
    if case["kind"] == "draw":
        return {"bytes": graph + 16 * n, "flops": 0}
    k, c = case["k"], case["c"]
    return {"bytes": graph + 8 * n * c, "flops": 2 * nnz * k + n * k * (2 * k + k + 2 * c)}


# ------------------------------------------------------------------------------------------------
# The layout in 64 bits with plain torch.

def _one_column(off, adj, src, w, source):
    n = off.numel() - 1
    if w is None:
        d = torch.full((n,), -1, dtype=torch.int64, device=off.device)
        d[source] = 0
        level, front = 0, torch.tensor([source], device=off.device)
        while front.numel():
            level += 1
            cnt = off[front + 1] - off[front]
            who = torch.repeat_interleave(torch.arange(front.numel(), device=off.device), cnt)
            e = torch.arange(who.numel(), device=off.device) - (torch.cumsum(cnt, 0) - cnt)[who] + off[front][who]
            front = adj[e]
            front = torch.unique(front[d[front] < 0])
            d[front] = level
        return d
    d = torch.full((n,), 1 << 40, dtype=torch.int64, device=off.device)
    d[source] = 0
    while True:
        for _ in range(8):
            nd = d.scatter_reduce(0, src, d[adj] + w, "amin")
            last, d = d, nd
        if torch.equal(last, d):
            return d


def _power(K):
    """Simultaneous power iteration from the C library's rand() stream, as the reference's solver runs it."""
    N = K.shape[0]
    r = [1]
    for _ in range(30):
        r.append(16807 * r[-1] % 2147483647)
    r += r[0:3]
    for i in range(34, N * N + 344):
        r.append((r[i - 31] + r[i - 3]) & 0xffffffff)
    E = np.array([x >> 1 for x in r[344:]], dtype=np.float64).reshape(N, N).T / 2147483647.0
    E = E / np.sqrt((E * E).sum(0))
    for _ in range(20000):
        T = E
        E = K @ T
        for i in range(1, N):
            for j in range(i):
                E[:, i] -= (E[:, j] @ E[:, i]) / (E[:, j] @ E[:, j]) * E[:, j]
        E = E / np.sqrt((E * E).sum(0))
        if np.abs((E * T).sum(0)).min() >= 1.0 - 1e-3:
            break
    out = np.empty_like(E)
    for j in range(N):  # ascending; the sign follows the first entry of the mirrored column
        out[:, j] = -E[:, N - 1 - j] if E[0, j] < 0 else E[:, N - 1 - j]
    return out


def _vectors(M, eig):
    M = M.cpu().numpy()
    if eig == "power":
        return _power(M)
    V = np.linalg.eigh((M + M.T) / 2)[1]
    return V * np.sign(V[np.abs(V).argmax(0), np.arange(V.shape[1])])


def exact(case, seed):
    if case["kind"] != "layout" or case["strategy"] != "Kcenters":
        return None
    if case["algo"] == "PivotMDS" and case["eig"] == "power":
        return None  # double centring leaves C^T C singular: the sweep at which the iteration stops is rounding's
    n, nnz = _size(case)
    k, c, hde = case["k"], case["c"], case["algo"] in ("ParHDE", "wParHDE")
    P = 3 * k if hde else k
    diameter = {"mesh": 2.0 * max(case.get("nx", 1), case.get("ny", 1)), "rmat": 8.0,
                "rgg2d": 1.2 * n ** 0.5, "rgg3d": 2.2 * n ** (1 / 3), "grid": 400.0 + 2.0 * n ** (1 / 3)}[case["graph"]]
    if (k + 2 if case["graph"] == "grid" else P) * (diameter * 3e-4 + nnz * (2e-9 if case["graph"] != "grid" else 1e-10 * diameter)) + k * nnz * 1e-9 > 12:
        return None
    off, adj, w = _graph(case, seed)[:3]
    n, src = off.numel() - 1, _rows(off)
    wl = None if w is None else w.long()
    deg = (off[1:] - off[:-1]).double() if w is None else torch.zeros(n, dtype=torch.float64, device=off.device).index_add(0, src, wl.double())
    least = torch.full((n,), 1 << 40, dtype=torch.int64, device=off.device)
    coupled = case["algo"] == "wParHDE"
    U = [torch.full((n,), n ** -0.5, dtype=torch.float64, device=off.device)]
    sources, history, cols, at = [], [], [], 0
    for p in range(P):
        d = _one_column(off, adj, src, wl, at)
        sources.append(at)
        least = torch.minimum(least, d)
        raw = nxt = int((least == least.max()).nonzero()[0])
        if (len(U) != 1 if coupled else p != 0) and raw in history:
            far = [v for v in (least == least.max()).nonzero()[:, 0].tolist() if v not in set(history)]
            nxt = far[-1] if far else raw
        history.append(raw if hde else at)
        at = nxt
        if not hde:
            cols.append(d.double())
            continue
        if len(U) > k:
            if coupled:
                sources.pop()
                break
            continue
        x = d.double()
        x = x / x.square().sum().sqrt()
        for again in range(2):  # twice: in exact arithmetic the second pass changes nothing
            for q in U:
                x = x - (x @ (deg * q)) / (q @ (deg * q)) * q
        norm = float(x.square().sum().sqrt())
        if norm >= 0.001:
            U.append(x / norm)
        if coupled and len(U) > k:
            break
    if not hde:
        C = torch.stack(cols, 1)
        if case["algo"] == "PivotMDS":
            C = C * C
            C = -0.5 * (C - C.mean(0) - C.mean(1, keepdim=True) + C.mean())
        else:
            C = C - C.mean(0)
        V = _vectors(C.T @ C, case["eig"])[:, ::-1]
        S = C
    else:
        if len(U) <= k:
            return None
        S = torch.stack(U[1:], 1)
        LS = deg[:, None] * S
        ww = None if w is None else w.double()
        for q in range(k):
            g = S[:, q][adj]
            LS[:, q].index_add_(0, src, -g if ww is None else -ww * g)
        V = _vectors(S.T @ LS, case["eig"])
    X = S @ torch.from_numpy(np.ascontiguousarray(V[:, :c])).to(S.device)
    X = X / X.square().sum(0).sqrt()
    return {"coords": X, "sources": torch.tensor(sources)}

"""Performance cases of the B200 traversal engine: the applications of
graphgrind_b200 (and one edgeMap step on device-resident vectors), each called
the way a program calls it through the C ABI: the graph is built once, results
go to page-locked host arrays that the program keeps.

Every kind of case covers a range of graph sizes (RANGES); listed() holds one
or two sizes of each, draw() gives others.  Graphs are random: R-MAT
(a, b, c, d) = (0.57, 0.19, 0.19, 0.05), Erdos-Renyi, or a 2D grid with 0.1 %
random long-range edges, without self-loops and duplicates, made from the seed
on the GPU; R-MAT vertex counts need not be powers of two (samples past n are
dropped).
"""
import ctypes as C
import math

import numpy as np
import torch

import graphgrind_b200 as gg

A, B, CC = 0.57, 0.19, 0.19  # R-MAT quadrant probabilities
DAMPING = 0.85

# kind -> vertices of the smallest and the largest case
RANGES = {
    "bfs": (1 << 10, 1 << 22),
    "bfs_grid": (64 * 64, 2049 * 2049),
    "components": (1 << 12, 1_000_003),
    "pagerank": (1 << 14, 1 << 22),
    "pagerank_delta": (1 << 14, 1 << 20),
    "spmv": (10_007, 1_500_007),
    "bellman_ford": (1 << 12, 1 << 20),
    "bc": (1 << 12, 700_001),
    "ppr": (1 << 12, 1 << 18),
    "batch": (1 << 10, 1 << 16),  # of one graph of the batch
    "weighted_pagerank": (1 << 12, 1 << 20),
}


def _case(kind, **kw):
    c = dict(kind=kind, graph="rmat", n=0, edge_factor=16, symmetric=False, partitions=384, hot_first=False,
             tile_edges=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a service answering one BFS at a time on a small
        # social graph, where launches and host round trips are all there is
        _case("bfs", name="bfs_rmat10", n=1 << 10, symmetric=True, partitions=16),
        # the headline traversal at a size where frontiers turn dense: directed
        # R-MAT, renumbered hottest-first as the benchmark builds its graph
        _case("bfs", name="bfs_rmat22", n=1 << 22, hot_first=True, tile_edges=1 << 18),
        # high diameter, sparse frontiers: road-like grid with an odd side
        _case("bfs_grid", name="bfs_grid2049", graph="grid", n=2049 * 2049, edge_factor=4, symmetric=True),
        # connected components of a symmetric graph of ragged size
        _case("components", name="components_1m", n=1_000_003, symmetric=True),
        # the headline ranking run: ten FP32 iterations on the benchmark's build
        _case("pagerank", name="pagerank_rmat22", n=1 << 22, hot_first=True, tile_edges=1 << 18),
        # incremental ranking until its change falls below 1e-7
        _case("pagerank_delta", name="pagerank_delta_rmat20", n=1 << 20),
        # one step of an iterative solver: y = A^T x with FP32 weights, vectors
        # resident on the device, no skew in the degrees
        _case("spmv", name="spmv_er_1m5", graph="er", n=1_500_007),
        # shortest paths with integer edge lengths in [1, 100]
        _case("bellman_ford", name="bellman_ford_rmat20", n=1 << 20),
        # betweenness contributions of one source, forward and backward
        _case("bc", name="bc_700k", n=700_001, symmetric=True),
        # 64 users' personalised rankings in one call
        _case("ppr", name="ppr64_rmat18", n=1 << 18, k=64, iters=20),
        # a collection of uneven graphs traversed in one call
        _case("batch", name="batch_256", n=1 << 16, graphs=256, edge_factor=32),
        # a training step on edge weights: forward and gradients
        _case("weighted_pagerank", name="weighted_pagerank_rmat20", n=1 << 20, edges=12 << 20, iters=30, every=5),
    ]


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    n = min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))
    parts = 384 if n >= 1 << 18 else 16 if n < 1 << 14 else 64
    if kind == "bfs":
        sym = rng.random() < 0.5
        return _case(kind, graph=rng.choice(["rmat", "rmat", "er"]), n=n // 2 if sym and n > 2048 else n,
                     symmetric=sym, partitions=parts, hot_first=rng.random() < 0.5)
    if kind == "bfs_grid":
        side = int(math.isqrt(n))
        return _case(kind, graph="grid", n=side * side, edge_factor=4, symmetric=True, partitions=parts)
    if kind in ("components", "bc"):
        return _case(kind, n=n, symmetric=True, partitions=parts, edge_factor=rng.choice([8, 16]))
    if kind == "pagerank":
        return _case(kind, graph=rng.choice(["rmat", "rmat", "er"]), n=n, partitions=parts,
                     hot_first=rng.random() < 0.5)
    if kind in ("pagerank_delta", "bellman_ford"):
        return _case(kind, n=n, partitions=parts, edge_factor=rng.choice([8, 16]))
    if kind == "spmv":
        return _case(kind, graph=rng.choice(["rmat", "er"]), n=n, partitions=parts)
    if kind == "ppr":
        return _case(kind, n=n, partitions=parts, k=rng.choice([32, 64]), iters=20)
    if kind == "batch":
        return _case(kind, n=max(n, 1 << 11), graphs=rng.randrange(16, 257), edge_factor=32)
    return _case(kind, n=n, edges=rng.randrange(6 * n, 12 * n), partitions=parts, iters=rng.choice([10, 30]), every=5)


# ------------------------------------------------------------------ graphs
def _gen(seed, salt):
    return torch.Generator("cuda").manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFF)


def _edge_keys(graph, n, edge_factor, symmetric, g):
    """Sorted distinct keys src * n + dst on the GPU."""
    cnt = n * edge_factor
    if graph == "rmat":
        src = torch.zeros(cnt, dtype=torch.int64, device="cuda")
        dst = torch.zeros_like(src)
        for _ in range(max(1, (n - 1).bit_length())):
            u = torch.rand(cnt, device="cuda", generator=g)
            low = u >= A + B
            src = src * 2 + low
            dst = dst * 2 + torch.where(low, u >= A + B + CC, u >= A)
        keep = (src < n) & (dst < n) & (src != dst)
        src, dst = src[keep], dst[keep]
    elif graph == "er":
        src = torch.randint(0, n, (cnt,), device="cuda", generator=g)
        dst = torch.randint(0, n, (cnt,), device="cuda", generator=g)
        keep = src != dst
        src, dst = src[keep], dst[keep]
    else:  # grid: right and down neighbours, then 0.1 % long-range edges
        side = math.isqrt(n)
        v = torch.arange(n, device="cuda")
        right, down = v[v % side != side - 1], v[v < n - side]
        extra = max(1, (2 * n) // 1000)
        a = torch.randint(0, n, (extra,), device="cuda", generator=g)
        b = torch.randint(0, n, (extra,), device="cuda", generator=g)
        keep = a != b
        src = torch.cat([right, down, a[keep]])
        dst = torch.cat([right + 1, down + side, b[keep]])
    key = src * n + dst
    if symmetric:
        key = torch.cat([key, dst * n + src])
    return torch.unique(key)


def _csr(graph, n, edge_factor, symmetric, g, edges=0):
    """(out-offsets, destinations, sources) as int64 tensors on the GPU; exactly `edges` random edges if given."""
    key = _edge_keys(graph, n, edge_factor, symmetric, g)
    if edges:
        while len(key) < edges:
            key = torch.unique(torch.cat([key, _edge_keys(graph, n, edge_factor, symmetric, g)]))
        key = key[torch.sort(torch.randperm(len(key), device="cuda", generator=g)[:edges])[0]]
    src = torch.div(key, n, rounding_mode="floor")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return off, key - src * n, src


def _case_csr(case, seed):
    return _csr(case["graph"], case["n"], case["edge_factor"], case["symmetric"], _gen(seed, 1), case.get("edges", 0))


def _u32(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


class _HostCsr:
    """A program's own CSR arrays as a gg_host_graph."""

    def __init__(self, off, dst, symmetric, weights=None):
        self.offsets, self.indices, self.weights = _u32(off), _u32(dst), weights
        self.n, self.m, self.symmetric = len(self.offsets) - 1, len(self.indices), bool(symmetric)
        wt = gg.W_NONE if weights is None else gg.W_FLOAT32 if weights.dtype == np.float32 else gg.W_INT32
        p = C.POINTER(C.c_uint32)
        self.c = gg.HostGraphC(self.n, self.m, int(symmetric), wt, self.offsets.ctypes.data_as(p),
                               self.indices.ctypes.data_as(p),
                               C.c_void_p(None if weights is None else weights.ctypes.data))


def _partitions(off, dst, n, m, preferred):
    """The largest of a few partition counts that the edge-balanced partitioner takes."""
    outd, ind = _u32(off[1:] - off[:-1]), _u32(torch.bincount(dst, minlength=n))
    for p in (384, 320, 256, 192, 128, 96, 64, 48, 32, 24, 16, 12, 8, 6, 4, 3, 2, 1):
        if p <= preferred:
            try:
                gg.partition_sizes(ind, outd, m, p)
                return p
            except gg.GGError:
                pass
    raise RuntimeError("no partition count accepted")


def _float_weights(m, seed):
    return 1 - torch.rand(m, device="cuda", generator=_gen(seed, 2))  # (0, 1]


def _int_weights(m, seed):
    return torch.randint(1, 101, (m,), device="cuda", generator=_gen(seed, 3))


def _vector(n, seed):
    return torch.rand(n, device="cuda", generator=_gen(seed, 4)) + 0.5


def _teleport(n, seed):
    t = _vector(n, seed)
    return t / t.sum()


def _loss_weights(n, seed):
    return torch.randn(n, device="cuda", generator=_gen(seed, 5))


def _ppr_seeds(n, k, seed):
    return torch.randint(0, n, (k,), device="cuda", generator=_gen(seed, 6))


def _start(off):
    """The first vertex from id 100 (or the middle of a smaller graph) with out-edges."""
    n = len(off) - 1
    deg = off[1:] - off[:-1]
    first = min(100, n // 2)
    return first + int(torch.nonzero(deg[first:])[0])


# ------------------------------------------------------------------- cases
class _DeviceView:
    """A library vertex array as something torch can wrap without a copy."""

    def __init__(self, arr, n):
        self.arr = arr
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (arr.ptr.value, False), "version": 3}


def _prepare_batch(case, seed):
    rng = np.random.default_rng(case["graphs"])  # the sizes are the case's, the graphs the seed's
    top = (case["n"] - 1).bit_length()
    hosts = []
    for i in range(case["graphs"]):
        n = 1 << int(rng.integers(10, top + 1))
        ef = int(rng.integers(8, case["edge_factor"] + 1))
        off, dst, _ = _csr("rmat", n, ef, False, _gen(seed, 100 + i))
        hosts.append(_HostCsr(off, dst, False))
    b = gg.GraphBatch(hosts)
    return dict(kind="batch", batch=b, sources=np.zeros(case["graphs"], np.uint32),
                out=gg.PinnedArray(b.total_vertices, np.int32))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    off, dst, _ = _case_csr(case, seed)
    n, m = case["n"], len(dst)
    weights = None
    if kind == "spmv":
        weights = _float_weights(m, seed).cpu().numpy()
    elif kind == "bellman_ford":
        weights = _int_weights(m, seed).to(torch.int32).cpu().numpy()
    host = _HostCsr(off, dst, case["symmetric"], weights)
    g = gg.Graph(host, partitions=_partitions(off, dst, n, m, case["partitions"]), tile_edges=case["tile_edges"],
                 vertex_order=gg.VORDER_HOT_FIRST if case["hot_first"] else gg.VORDER_GIVEN)
    s = dict(kind=kind, graph=g, stats=gg.RunStats())
    if kind in ("bfs", "bfs_grid", "bellman_ford"):
        s.update(start=_start(off), out=gg.PinnedArray(n, np.int32))
    elif kind == "components":
        s.update(out=gg.PinnedArray(n, np.int32))
    elif kind in ("pagerank", "pagerank_delta"):
        s.update(out=gg.PinnedArray(n, np.float32))
    elif kind == "bc":
        s.update(start=_start(off), dep=gg.PinnedArray(n, np.float32), paths=gg.PinnedArray(n, np.float32))
    elif kind == "ppr":
        s.update(k=case["k"], iters=case["iters"], seeds=_u32(_ppr_seeds(n, case["k"], seed)),
                 out=gg.PinnedArray(n * case["k"], np.float32))
    elif kind == "spmv":
        x, y = gg.DeviceArray(g, np.float32), gg.DeviceArray(g, np.float32)
        x.upload(_vector(n, seed).cpu().numpy())
        fill = (C.c_double * 2)()  # gg_fill_args {array, value = 0}
        C.cast(fill, C.POINTER(C.c_void_p))[0] = y.ptr
        s.update(all=g.frontier_all(), args=gg.PairArgs(x.ptr, y.ptr), fill=fill, x=x,
                 y=torch.as_tensor(_DeviceView(y, n), device="cuda"), y_array=y)
    else:
        def pinned(t):
            p = gg.PinnedArray(len(t), np.float32)
            p.array[:] = t.cpu().numpy()
            return p
        s.update(wpr=gg.WeightedPageRank(g, iters=case["iters"], damping=DAMPING, checkpoint_every=case["every"],
                                         normalize=True),
                 w=pinned(_float_weights(m, seed)), tele=pinned(_teleport(n, seed)),
                 grad=pinned(_loss_weights(n, seed)), x=gg.PinnedArray(n, np.float32),
                 gw=gg.PinnedArray(m, np.float32), gt=gg.PinnedArray(n, np.float32),
                 g0=gg.PinnedArray(n, np.float32))
    return s


FILL_F32 = 103  # GG_V_FILL_F32


def run(s):
    lib, kind = gg.lib, s["kind"]
    if kind == "batch":
        return s["batch"].bfs(s["sources"], s["out"].array)[0]
    g, st = s["graph"], C.byref(s["stats"])
    if kind in ("bfs", "bfs_grid"):  # levels alone: any tree of parents would do
        gg.check(lib.gg_bfs(g.h, s["start"], None, s["out"].ptr, st), "gg_bfs")
        return s["out"].array
    if kind == "components":
        gg.check(lib.gg_components(g.h, s["out"].ptr, st), "gg_components")
        return s["out"].array
    if kind == "pagerank":
        return g.pagerank(10, out=s["out"].array)[0]
    if kind == "pagerank_delta":
        gg.check(lib.gg_pagerank_delta(g.h, s["out"].ptr, st), "gg_pagerank_delta")
        return s["out"].array
    if kind == "bellman_ford":
        gg.check(lib.gg_bellman_ford(g.h, s["start"], s["out"].ptr, st), "gg_bellman_ford")
        return s["out"].array
    if kind == "bc":
        gg.check(lib.gg_bc(g.h, s["start"], s["dep"].ptr, s["paths"].ptr, st), "gg_bc")
        return s["dep"].array, s["paths"].array
    if kind == "ppr":
        return g.ppr_k(s["k"], s["iters"], DAMPING, seeds=s["seeds"], out=s["out"].array)[0]
    if kind == "spmv":
        gg.check(lib.gg_vertex_map(g.h, s["all"].h, FILL_F32, C.cast(s["fill"], C.c_void_p)), "gg_vertex_map")
        g.edge_map(s["all"], gg.F_SPMV, s["args"], flags=gg.EM_NO_OUTPUT).close()
        return s["y"]
    h = s["wpr"].h
    gg.check(lib.gg_pagerank_weighted_fwd(h, s["w"].ptr, s["tele"].ptr, None, s["x"].ptr, st), "forward")
    gg.check(lib.gg_pagerank_weighted_bwd(h, s["grad"].ptr, s["gw"].ptr, s["gt"].ptr, s["g0"].ptr, st), "backward")
    return s["x"].array, s["gw"].array, s["gt"].array, s["g0"].array


def work(case):
    """Edges as 4-byte ids (and weights) read once a pass over them, vertex values read and written once."""
    kind, n = case["kind"], case["n"]
    m = case.get("edges") or n * case["edge_factor"] * (2 if case["symmetric"] else 1)
    if kind == "batch":  # scales and edge factors are uniform
        top = (n - 1).bit_length()
        mean_n = sum(1 << s for s in range(10, top + 1)) / (top - 9)
        mean_ef = (8 + case["edge_factor"]) / 2
        return {"bytes": case["graphs"] * mean_n * (4 * mean_ef + 8), "flops": 0}
    if kind in ("bfs", "bfs_grid", "components"):
        return {"bytes": 4 * m + 8 * n, "flops": 0}
    if kind == "pagerank":
        return {"bytes": 10 * (4 * m + 12 * n), "flops": 10 * 2 * m}
    if kind == "pagerank_delta":
        return {"bytes": 4 * m + 16 * n, "flops": 2 * m}
    if kind == "spmv":
        return {"bytes": 8 * m + 12 * n, "flops": 2 * m}
    if kind == "bellman_ford":
        return {"bytes": 8 * m + 8 * n, "flops": 0}
    if kind == "bc":
        return {"bytes": 2 * (4 * m + 12 * n), "flops": 2 * m}
    if kind == "ppr":
        return {"bytes": case["iters"] * (4 * m + 8 * n * case["k"]), "flops": case["iters"] * 2 * m * case["k"]}
    it = case["iters"]
    return {"bytes": it * (8 * m + 12 * n) + it * (12 * m + 16 * n), "flops": it * 6 * m}


# ---------------------------------------------------------- 64-bit results
def _gather_sum(src, dst, val, n):
    """sum over edges of val[src], at dst."""
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dst, val[src])


def _inv_degree(off):
    deg = (off[1:] - off[:-1]).double()
    return torch.where(deg > 0, 1 / deg, torch.zeros_like(deg))


def _exact_pagerank(off, dst, src, n):
    inv, added = _inv_degree(off), (1 - DAMPING) / n
    p = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    acc = torch.zeros_like(p)
    member = torch.ones(n, dtype=torch.bool, device="cuda")
    for _ in range(10):
        contrib = torch.where(member, p * inv, torch.zeros_like(p))
        touched = _gather_sum(src, dst, member.double(), n) > 0
        nxt = acc + _gather_sum(src, dst, contrib, n)
        nxt = torch.where(member, DAMPING * nxt + added, nxt)
        diff = (p - nxt).abs()
        acc = torch.where(member, torch.zeros_like(diff), diff)
        p, member = nxt, touched
        if float(diff.sum()) < 1e-7:
            break
    return p


def _exact_pagerank_delta(off, dst, src, n):
    inv, added = _inv_degree(off), (1 - DAMPING) / n
    p = torch.zeros(n, dtype=torch.float64, device="cuda")
    delta = torch.full_like(p, 1.0 / n)
    member = torch.ones(n, dtype=torch.bool, device="cuda")
    for r in range(1000):
        ngh = _gather_sum(src, dst, torch.where(member, delta * inv, torch.zeros_like(p)), n)
        if r == 0:
            d = DAMPING * (p + ngh) + added - p
            p = p + d
            d = d - 1.0 / n
        else:
            d = DAMPING * ngh
            p = p + d
        delta, member = d, d.abs() > 0.01 * p
        if float(delta.abs().sum()) < 1e-7:
            break
    return p


def _exact_bc(off, dst, src, n, start):
    level = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    paths = torch.zeros(n, dtype=torch.float64, device="cuda")
    level[start], paths[start], last = 0, 1.0, 0
    while True:
        on = level[src] == last
        fresh = on & (level[dst] < 0)
        if not bool(fresh.any()):
            break
        paths.index_add_(0, dst[fresh], paths[src[fresh]])
        last += 1
        level[dst[fresh]] = last
    inv = 1 / paths
    dep = torch.where(level == last, inv, torch.zeros_like(inv))
    for r in range(last - 1, -1, -1):
        succ = (level[src] == r) & (level[dst] == r + 1)
        dep.index_add_(0, src[succ], dep[dst[succ]])
        dep = torch.where(level == r, dep + inv, dep)
    return (dep - inv) / inv, paths


def _exact_ppr(off, dst, src, n, k, iters, seeds):
    tele = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    tele[seeds, torch.arange(k, device="cuda")] = 1.0
    adj = torch.sparse_coo_tensor(torch.stack([dst, src]), _inv_degree(off)[src], (n, n)).to_sparse_csr()
    x = tele
    for _ in range(iters):
        x = DAMPING * (adj @ x) + (1 - DAMPING) * tele
    return x


def _exact_weighted(off, dst, src, n, w, tele, grad, iters):
    wsum = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, src, w)
    a = w / wsum[src]
    xs = [torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")]
    for _ in range(iters):
        s = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dst, a * xs[-1][src])
        xs.append(DAMPING * s + (1 - DAMPING) * tele)
    lam, ga, gt = grad, torch.zeros_like(a), torch.zeros_like(tele)
    for t in range(iters - 1, -1, -1):
        gt = gt + (1 - DAMPING) * lam
        back = lam[dst]
        ga += DAMPING * back * xs[t][src]
        lam = DAMPING * torch.zeros_like(gt).index_add_(0, src, a * back)
    r = torch.zeros_like(wsum).index_add_(0, src, ga * a)
    return xs[-1], (ga - r[src]) / wsum[src], gt, lam


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("bfs", "bfs_grid", "components", "bellman_ford", "batch"):
        return None  # whole numbers
    off, dst, src = _case_csr(case, seed)
    if kind == "pagerank":
        return _exact_pagerank(off, dst, src, n)
    if kind == "pagerank_delta":
        return _exact_pagerank_delta(off, dst, src, n)
    if kind == "spmv":
        y = torch.zeros(n, dtype=torch.float64, device="cuda")
        return y.index_add_(0, dst, _vector(n, seed).double()[src] * _float_weights(len(dst), seed).double())
    if kind == "bc":
        return _exact_bc(off, dst, src, n, _start(off))
    if kind == "ppr":
        return _exact_ppr(off, dst, src, n, case["k"], case["iters"], _ppr_seeds(n, case["k"], seed))
    return _exact_weighted(off, dst, src, n, _float_weights(len(dst), seed).double(), _teleport(n, seed).double(),
                           _loss_weights(n, seed).double(), case["iters"])

"""The performance cases of this framework: what its users have it do.

A case is one call sequence of an analytics program over a multiversion graph
(benchmark tasks of LLAMA over a snapshot of a level stack), on a seeded
synthetic graph made on the GPU: R-MAT (a, b, c = .57, .19, .19) or a
scrambled symmetric Kronecker graph, split over several levels with deletion
marks, as the benchmark's own workloads are.  Vertex counts are not powers of
two unless a case stands for the benchmark's own graph.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  store, snapshot and buffers a program holds
  run(state)           one pass through the public entry points
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    the floating results by plain torch in 64 bits
"""
import math

import numpy as np
import torch

from llama_b200 import Store
from llama_b200.graph import ppr

A, B, C = 0.57, 0.19, 0.19
DAMPING = 0.85

# Ranges per task: vertices (log2), edge factor, and the task's own options.
RANGES = {
    "step": dict(lg_v=(12, 24), ef=(8, 16), levels=(1, 8), iters=(5, 20), roots=(2, 16)),
    "pagerank": dict(lg_v=(11, 22), ef=(4, 24), levels=(1, 8), iters=(5, 20)),
    "push": dict(lg_v=(11, 21), ef=(4, 20), levels=(1, 8), iters=(5, 20)),
    "bfs": dict(lg_v=(11, 23), ef=(4, 20), levels=(1, 8)),
    "sssp": dict(lg_v=(11, 22), ef=(4, 20), levels=(1, 8), delta=(8, 64)),
    "scc": dict(lg_v=(11, 22), ef=(4, 20), levels=(1, 8)),
    "triangles": dict(lg_v=(10, 19.5), ef=(4, 16), levels=(1, 4)),
    "bc": dict(lg_v=(10, 18), ef=(4, 20), levels=(1, 4), sources=(1, 128)),
    "ppr": dict(lg_v=(10, 17), ef=(4, 20), levels=(1, 4), iters=(5, 20)),
    "adjoint": dict(lg_v=(10, 19), ef=(4, 20), levels=(1, 8)),
    "update": dict(lg_v=(12, 22), ef=(8, 16), levels=(2, 8), iters=(2, 5)),
}
# vertices x arcs per vertex x seeds x snapshots x iterations of a drawn
# personalised PageRank: no more than two thirds of the listed one's
PPR_MOST = 9_000_000_000


def _case(task, V, ef, levels, **more):
    c = dict(task=task, V=int(V), ef=int(ef), levels=int(levels), kind="rmat", delete=0.002,
             flat=False)
    c.update(more)
    return c


def listed():
    return [
        # an interactive query on a small graph, result wanted on the host:
        # launches and copies count, not bandwidth
        dict(name="pagerank_small_host",
             **_case("pagerank", 3001, 8, 2, iters=10, host=True)),
        # a PageRank job on a snapshot nobody flattened, odd sizes
        dict(name="pagerank_1m", **_case("pagerank", 1000003, 14, 4, iters=20, host=False)),
        # the benchmark's own step: flatten, 20 iterations, BFS from 16 roots
        dict(name="step_rmat24", **_case("step", 1 << 24, 16, 8, iters=20, roots=16)),
        # PageRank where a store is kept without reverse edges
        dict(name="push_2m", **_case("push", 1900001, 12, 4, iters=10)),
        # single queries: hop distances, weighted distances (flattened graphs)
        dict(name="bfs_4m", **_case("bfs", 4000037, 16, 8, flat=True)),
        dict(name="sssp_3m", **_case("sssp", 3000017, 16, 4, flat=True, delta=32)),
        # structure of a directed graph: components, triangles
        dict(name="scc_3m", **_case("scc", 3000017, 14, 4)),
        dict(name="triangles_700k", **_case("triangles", 700001, 16, 4)),
        # centrality of an undirected graph from a ragged batch of sources
        dict(name="bc_200k", **_case("bc", 200003, 16, 4, kind="kron", delete=0.0, sources=80)),
        # personalised PageRank for a batch of seeds on successive snapshots
        dict(name="ppr_100k",
             **_case("ppr", 100003, 16, 4, kind="kron", delete=0.0, iters=15, seeds=96, snaps=3)),
        # learning edge weights: forward to the fixed point and its gradients
        dict(name="adjoint_250k", **_case("adjoint", 250007, 16, 4)),
        # a checkpoint arrives from the host and the ranks are refreshed
        dict(name="update_3m", **_case("update", 3000017, 16, 8, iters=3)),
    ]


def draw(rng):
    task = rng.choice(sorted(RANGES))
    r = RANGES[task]
    V = int(2.0 ** rng.uniform(*r["lg_v"]))
    if rng.random() < 0.6:
        V |= 1
    ef = int(round(math.exp(rng.uniform(math.log(r["ef"][0]), math.log(r["ef"][1])))))
    c = _case(task, V, ef, rng.randint(*r["levels"]), delete=rng.choice([0.0, 0.002, 0.01]))
    if task in ("triangles", "bc", "ppr") and rng.random() < 0.6:
        c["kind"], c["delete"] = "kron", 0.0
    if "iters" in r:
        c["iters"] = rng.randint(*r["iters"])
    if "roots" in r:
        c["roots"] = rng.randint(*r["roots"])
    if task == "pagerank":
        c["host"] = V < 65536 and rng.random() < 0.5
    if task in ("pagerank", "push", "bfs", "sssp"):
        c["flat"] = rng.random() < 0.5
    if task == "sssp":
        c["delta"] = rng.randint(*r["delta"])
    if task == "bc":
        c["sources"] = rng.randint(*r["sources"])
    if task == "ppr":
        c["seeds"] = 32 * rng.randint(1, 4)
        c["snaps"] = rng.randint(1, c["levels"])
        arcs = ef * (2 if c["kind"] == "kron" else 1)
        most = PPR_MOST // (arcs * c["seeds"] * c["snaps"] * c["iters"])
        c["V"] = min(c["V"], most)
    return c


# ---------------------------------------------------------------------------
# Graphs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7fffffff)
    return g


class Edges:
    """Distinct edges sorted by (src, dst), the level each was added in, and
    the level that deleted it (number of levels = never)."""

    def __init__(self, case, seed):
        self.V, self.L = case["V"], case["levels"]
        g = self.gen = _gen(seed)
        kron = case["kind"] == "kron"
        bits = max(1, (self.V - 1).bit_length())
        todo, keys = self.V * case["ef"], []
        while todo > 0:
            n = min(todo, 1 << 25)
            todo -= n
            s = torch.zeros(n, dtype=torch.int32, device="cuda")
            d = torch.zeros(n, dtype=torch.int32, device="cuda")
            for _ in range(bits):
                u = torch.rand(n, generator=g, device="cuda")
                lo = u >= A + B
                s.mul_(2).add_(lo)
                d.mul_(2).add_(((u >= A) & ~lo) | (u >= A + B + C))
            ok = (s < self.V) & (d < self.V) & (s != d)
            s, d = s[ok].long(), d[ok].long()
            if kron:
                s, d = torch.minimum(s, d), torch.maximum(s, d)
            keys.append((s << 32) | d)
        key = torch.unique(torch.cat(keys))
        del keys
        n = key.numel()
        f0 = 1.0 / self.L if kron else 0.9
        u = torch.rand(n, generator=g, device="cuda")
        lev = torch.zeros(n, dtype=torch.int8, device="cuda")
        if self.L > 1:
            lev = (1 + (u - f0) * ((self.L - 1) / (1 - f0))).floor().clamp_(0, self.L - 1)
            lev = torch.where(u < f0, torch.zeros_like(lev), lev).to(torch.int8)
        src, dst = (key >> 32).int(), (key & 0xffffffff).int()
        del key, u
        if kron:                    # scrambled ids, both arcs of every edge
            p = torch.randperm(self.V, generator=g, device="cuda").int()
            src, dst = p[src.long()], p[dst.long()]
            src, dst, lev = torch.cat([src, dst]), torch.cat([dst, src]), torch.cat([lev, lev])
            o = torch.argsort((src.long() << 32) | dst.long())
            src, dst, lev = src[o], dst[o], lev[o]
        self.src, self.dst, self.lev = src, dst, lev
        self.death = torch.full_like(lev, self.L)
        if case["delete"] > 0:
            for l in range(1, self.L):
                hit = torch.rand(lev.numel(), generator=g, device="cuda") < case["delete"]
                self.death[hit & (lev < l) & (self.death == self.L)] = l

    def level(self, l):
        """(src, dst, del_src, del_dst) of level l."""
        new, dead = self.lev == l, self.death == l
        if l == 0:
            dead = torch.zeros_like(dead)
        return self.src[new], self.dst[new], self.src[dead], self.dst[dead]

    def live(self, l):
        """(src, dst) of the edges live in snapshot l, as int64."""
        m = (self.lev <= l) & (self.death > l)
        return self.src[m].long(), self.dst[m].long()

    def out_order(self):
        """Live edges of the newest snapshot in out-adjacency order: per
        vertex newest level first, by target inside a level."""
        m = self.death == self.L
        s, d, lev = self.src[m].long(), self.dst[m].long(), self.lev[m].long()
        o = torch.argsort(s * self.L + (self.L - 1 - lev), stable=True)
        return s[o], d[o]

    def sources(self, n):
        """n vertices with out-edges, drawn by degree (sources of live edges)."""
        s, _ = self.live(self.L - 1)
        at = torch.randint(0, s.numel(), (n,), generator=self.gen, device="cuda")
        return s[at].cpu().numpy()


class State:
    """What a program holds: the store, the snapshot and its buffers."""

    def __init__(self):
        self.snaps, self.store = [], None

    def __del__(self):
        for s in self.snaps:
            s.close()
        if self.store is not None:
            self.store.close()


def _adjoint_inputs(case, e):
    s, _ = e.out_order()
    deg = torch.bincount(s, minlength=e.V).double()
    w = (0.5 + 0.5 * torch.rand(s.numel(), generator=e.gen, device="cuda",
                                dtype=torch.float64)) / deg[s]
    v = torch.rand(e.V, generator=e.gen, device="cuda", dtype=torch.float64) / e.V
    g = torch.randn(e.V, generator=e.gen, device="cuda", dtype=torch.float64) / e.V
    return w, v, g


def prepare(case, seed):
    e = Edges(case, seed)
    st = State()
    st.case, V, L, task = case, case["V"], case["levels"], case["task"]
    st.store = Store(reverse_edges=task != "push")
    build = L - 1 if task == "update" else L
    for l in range(build):
        s, d, xs, xd = e.level(l)
        w = None
        if task == "sssp":
            w = torch.randint(1, 256, (s.numel(),), generator=e.gen, device="cuda",
                              dtype=torch.int32)
        torch.cuda.synchronize()
        st.store.build_level(V, s, d, w, xs, xd)
    if task == "update":
        s, d, xs, xd = e.level(L - 1)
        p = torch.randperm(s.numel(), generator=e.gen, device="cuda")
        st.delta = [x.cpu().numpy().view(np.uint32) for x in (s[p], d[p], xs, xd)]
    else:
        first = L - case["snaps"] if task == "ppr" else L - 1
        st.snaps = [st.store.snapshot(l) for l in range(first, L)]
    if case["flat"]:
        st.snaps[-1].flatten(1 if task in ("pagerank", "bfs") else 0)
    f64 = dict(dtype=torch.float64, device="cuda")
    if task in ("step", "pagerank", "push", "update"):
        st.ranks = None if case.get("host") else torch.empty(V, **f64)
    if task == "step":
        st.roots = e.sources(case["roots"])
        st.levels = torch.empty((case["roots"], V), dtype=torch.int32, device="cuda")
    elif task in ("bfs", "sssp"):
        st.root = int(e.sources(1)[0])
        st.dist = torch.empty(V, dtype=torch.int32, device="cuda")
    elif task == "scc":
        st.labels = torch.empty(V, dtype=torch.int64, device="cuda")
    elif task == "bc":
        st.sources = e.sources(case["sources"])
        st.bc = torch.empty(V, **f64)
    elif task == "ppr":
        st.seeds = e.sources(case["seeds"])
        st.x = torch.empty((case["snaps"], V, case["seeds"]), **f64)
    elif task == "adjoint":
        st.w, st.v, st.g = _adjoint_inputs(case, e)
        st.x, st.dv = torch.empty_like(st.v), torch.empty_like(st.v)
        # one length for every graph of a case; the edges there are come first
        st.dw = torch.zeros(case["ef"] * V * (2 if case["kind"] == "kron" else 1), **f64)
    del e
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return st


def run(st):
    c, task = st.case, st.case["task"]
    sn = st.snaps[-1] if st.snaps else None
    if task == "pagerank":
        return sn.pagerank_pull(c["iters"], DAMPING, out=st.ranks)
    if task == "push":
        return sn.pagerank_push(c["iters"], DAMPING, out=st.ranks)
    if task == "step":
        sn.flatten(1)
        sn.pagerank_pull(c["iters"], DAMPING, out=st.ranks)
        _, r = sn.bfs_multi(st.roots, out=st.levels)
        sn.unflatten()
        return {"ranks": st.ranks, "levels": st.levels, "reached": [int(x.reached) for x in r],
                "edges": [int(x.reach_edges) for x in r]}
    if task == "bfs":
        _, r = sn.bfs(st.root, out=st.dist)
        return {"levels": st.dist, "reached": int(r.reached), "edges": int(r.reach_edges),
                "depth": int(r.max_level)}
    if task == "sssp":
        _, r = sn.sssp(st.root, c["delta"], out=st.dist)
        return {"dist": st.dist, "reached": int(r.reached), "edges": int(r.reach_edges),
                "far": int(r.max_dist)}
    if task == "scc":
        _, r = sn.scc(out=st.labels)
        return {"labels": st.labels, "components": int(r.components)}
    if task == "triangles":
        r = sn.triangle_count()
        return {"triangles": int(r.triangles), "edges": int(r.undirected_edges),
                "arcs": int(r.arcs)}
    if task == "bc":
        return sn.bc(st.sources, out=st.bc)
    if task == "ppr":
        return ppr(st.snaps, st.seeds, c["iters"], DAMPING, out=st.x)
    if task == "adjoint":
        _, tape, _ = sn.pagerank_fwd(st.w, st.v, DAMPING, tol=1e-12, out=st.x)
        tape.backward(st.g, dldw=st.dw, dldv=st.dv)
        tape.close()
        return {"x": st.x, "dw": st.dw, "dv": st.dv}
    # update: the newest level from the host, the ranks of the new snapshot
    s, d, xs, xd = st.delta
    st.store.build_level(c["V"], s, d, None, xs, xd)
    with st.store.snapshot() as new:
        new.pagerank_pull(c["iters"], DAMPING, out=st.ranks)
        deg = new.out_degrees()
    st.store.drop_level()
    return {"ranks": st.ranks, "degrees": deg.view(np.int32)}


def work(case):
    """Each id, weight and vector element read once, each result written once
    per sweep the algorithm cannot do without (E estimated before the
    generator drops duplicates)."""
    V, t = case["V"], case["task"]
    E = 0.95 * case["ef"] * V * (2 if case["kind"] == "kron" else 1)
    sweep, n = 4 * E + 16 * V, case.get("iters", 1)
    if t in ("pagerank", "push"):
        return {"bytes": n * sweep, "flops": 2 * n * E}
    if t == "step":
        return {"bytes": 8 * E + n * sweep + 4 * E + 4 * V * case["roots"], "flops": 2 * n * E}
    if t == "update":
        return {"bytes": 8 * E + n * sweep + 16 * V, "flops": 2 * n * E}
    if t == "bfs":
        return {"bytes": 4 * E + 8 * V, "flops": E}
    if t == "sssp":
        return {"bytes": 8 * E + 8 * V, "flops": 2 * E}
    if t == "scc":
        return {"bytes": 8 * E + 16 * V, "flops": 2 * E}
    if t == "triangles":
        return {"bytes": 4 * E + 8 * V, "flops": E * case["ef"]}
    if t == "bc":
        s = case["sources"]
        return {"bytes": 8 * E + 24 * V * s, "flops": 4 * E * s}
    if t == "ppr":
        k, m = case["seeds"], case["snaps"]
        return {"bytes": m * n * (4 * E + 16 * V * k), "flops": 2 * m * n * E * k}
    its = 60                       # sweeps to 1e-12 and back, at the least
    return {"bytes": 2 * its * (12 * E + 24 * V) + 24 * E, "flops": 4 * its * E}


# ---------------------------------------------------------------------------
# The floating results in 64 bits
# ---------------------------------------------------------------------------

def _ranks(V, s, d, iters):
    deg = torch.bincount(s, minlength=V).double()
    x = torch.full((V,), 1.0 / V, dtype=torch.float64, device="cuda")
    for _ in range(iters):
        y = torch.where(deg > 0, x / deg, torch.zeros_like(x))
        acc = torch.zeros_like(x).index_add_(0, d, y[s])
        x = (1.0 - DAMPING) / V + DAMPING * acc
    return x


def _matrix(rows, cols, V, values=None):
    o = torch.argsort(rows * V + cols)
    off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=V), 0)
    val = torch.ones(rows.numel(), dtype=torch.float64, device="cuda") if values is None \
        else values[o]
    return torch.sparse_csr_tensor(off, cols[o], val, (V, V))


def _brandes(V, s, d, sources):
    out, into = _matrix(s, d, V), _matrix(d, s, V)
    bc = torch.zeros(V, dtype=torch.float64, device="cuda")
    for p in range(0, len(sources), 64):
        roots = torch.as_tensor(sources[p:p + 64], device="cuda")
        k = roots.numel()
        at = torch.arange(k, device="cuda")
        sigma = torch.zeros((V, k), dtype=torch.float64, device="cuda")
        depth = torch.full((V, k), -1, dtype=torch.int32, device="cuda")
        sigma[roots, at], depth[roots, at] = 1.0, 0
        top = 0
        while True:
            f = into @ torch.where(depth == top, sigma, torch.zeros_like(sigma))
            new = (f > 0) & (depth < 0)
            if not bool(new.any()):
                break
            top += 1
            sigma = torch.where(new, f, sigma)
            depth = depth.masked_fill(new, top)
        delta = torch.zeros_like(sigma)
        for l in range(top - 1, -1, -1):
            q = torch.where(depth == l + 1, (1.0 + delta) / sigma, torch.zeros_like(sigma))
            delta = torch.where(depth == l, sigma * (out @ q), delta)
        delta[roots, at] = 0.0
        bc += delta.sum(1)
    return bc


def _fixed_point(m, base, x):
    for _ in range(4000):
        y = base + DAMPING * (m @ x.unsqueeze(1)).squeeze(1)
        done = float((y - x).abs().sum()) < 1e-13 * max(1.0, float(y.abs().sum()))
        x = y
        if done:
            break
    return x


def exact(case, seed):
    task, V, L = case["task"], case["V"], case["levels"]
    if task in ("bfs", "sssp", "scc", "triangles"):
        return None                # whole numbers only
    e = Edges(case, seed)
    if task == "adjoint":
        s, d = e.out_order()
        w, v, g = _adjoint_inputs(case, e)
        x = _fixed_point(_matrix(d, s, V, w), (1.0 - DAMPING) * v, v)
        lam = _fixed_point(_matrix(s, d, V, w), g, g)
        dw = torch.zeros(case["ef"] * V * (2 if case["kind"] == "kron" else 1),
                         dtype=torch.float64, device="cuda")
        dw[:s.numel()] = DAMPING * lam[d] * x[s]
        return {"x": x, "dw": dw, "dv": (1.0 - DAMPING) * lam}
    if task == "ppr":
        # the seeds follow the level builds, which draw nothing
        seeds = torch.as_tensor(e.sources(case["seeds"]), device="cuda")
        at = torch.arange(seeds.numel(), device="cuda")
        xs = []
        for l in range(L - case["snaps"], L):
            s, d = e.live(l)
            deg = torch.bincount(s, minlength=V).double().unsqueeze(1)
            m = _matrix(d, s, V)
            x = torch.zeros((V, seeds.numel()), dtype=torch.float64, device="cuda")
            x[seeds, at] = 1.0
            for _ in range(case["iters"]):
                x = DAMPING * (m @ torch.where(deg > 0, x / deg, torch.zeros_like(x)))
                x[seeds, at] += 1.0 - DAMPING
            xs.append(x)
        return torch.stack(xs)
    s, d = e.live(L - 1)
    if task == "bc":
        return _brandes(V, s, d, e.sources(case["sources"]))
    ranks = _ranks(V, s, d, case["iters"])
    if task == "step":
        n = case["roots"]
        return {"ranks": ranks, "levels": None, "reached": [None] * n, "edges": [None] * n}
    if task == "update":
        return {"ranks": ranks, "degrees": None}
    return ranks

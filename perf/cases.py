"""Workloads of the traversal library, each one call (or one wave of requests) a user's program makes.

A case is a dict of plain values:
  kind      which entry point: "sssp", "ppr" (one query), "sssp_batch", "ppr_batch" (many sources in one
            call), "adsorption" (16 labels), "adjoint" (gradient of a PPR score by edge weight), "serve"
            (a wave of mixed requests to the serving loop)
  graph     "rmat" (a/b/c/d = 0.57/0.19/0.19/0.05, ids folded into [0, V)) or "uniform" random edges
  V, ef     vertices and drawn edges per vertex (self-loops and duplicate edges are removed; the adjoint,
            whose gradient has one entry per edge, gets exactly V * ef edges where the draw has as many)
  wmax      int32 weights are uniform in [1, wmax]; float weights are uniform, normalised per source
  pruned    the graph is pruned first (purn-sssp / purn-ppr) and each query starts from its own records
  n         sources per call: half uniform over vertices with out-edges, half from the top 1% out-degree
  host      results go to host arrays (the binding's default) instead of device memory
  alpha, rmax, iterations, targets: parameters of the push, the label propagation and the adjoint

prepare() holds what a program holds before the call: the resident graph handle (or server), the sources and,
for device results, the output buffers.
"""
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "c-2graph_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import c2g  # noqa: E402


def listed():
    return [
        # One shortest-path query on a graph of a few thousand vertices, result to the host: a call whose
        # time is launches, barriers and latency (the size of the repository's small parity graphs).
        dict(name="sssp-one-s12", kind="sssp", graph="rmat", V=4096, ef=8, wmax=100, pruned=False, n=1, host=True),
        # sssp-purn on the plain SSSP configuration: scale 16, pruned, the query's own records as seeds.
        dict(name="sssp-one-s16-pruned", kind="sssp", graph="rmat", V=65536, ef=16, wmax=100, pruned=True, n=1,
             host=True),
        # sssp-base on the single-query configuration: scale 22, result kept on the device.
        dict(name="sssp-one-s22", kind="sssp", graph="rmat", V=4194304, ef=16, wmax=1000, pruned=False, n=1,
             host=False),
        # ppr-base with the reference's default parameters on a small graph, result to the host.
        dict(name="ppr-one-s14", kind="ppr", graph="rmat", V=16384, ef=8, wmax=100, pruned=False, n=1, host=True,
             alpha=0.2, rmax=0.0),
        # ppr-base at the adjoint configuration's graph size with the serving parameters.
        dict(name="ppr-one-s20", kind="ppr", graph="rmat", V=1048576, ef=16, wmax=1000, pruned=False, n=1, host=False,
             alpha=0.15, rmax=1e-7),
        # A part-filled batch of one query word on a graph of the size of the reference's shipped web graph
        # (685,230 vertices, 7.6M edges), without hubs, distances to the host.
        dict(name="sssp-batch-31-web", kind="sssp_batch", graph="uniform", V=685230, ef=11, wmax=100, pruned=False,
             n=31, host=True),
        # The multi-tenant batch: 256 seeded shortest-path queries on the pruned scale-22 graph.
        dict(name="sssp-batch-256-s22", kind="sssp_batch", graph="rmat", V=4194304, ef=16, wmax=1000, pruned=True,
             n=256, host=False),
        # A small ragged PPR batch: 40 queries, two query words, the second part-filled.
        dict(name="ppr-batch-40-s16", kind="ppr_batch", graph="rmat", V=65536, ef=16, wmax=100, pruned=False, n=40,
             host=False, alpha=0.15, rmax=1e-7),
        # The multi-tenant PPR batch: 256 seeded queries on a pruned R-MAT graph.
        dict(name="ppr-batch-256-s21", kind="ppr_batch", graph="rmat", V=2097152, ef=16, wmax=1000, pruned=True,
             n=256, host=False, alpha=0.15, rmax=1e-7),
        # One label-propagation request: 16 labels, 30 iterations.
        dict(name="adsorption-s22", kind="adsorption", graph="rmat", V=4194304, ef=16, wmax=1000, pruned=False, n=1,
             host=False, iterations=30),
        # The adjoint configuration: 64 random targets, gradient of every edge weight to the host.
        dict(name="adjoint-s20", kind="adjoint", graph="rmat", V=1048576, ef=16, wmax=1000, pruned=False, n=1,
             host=True, alpha=0.15, rmax=1e-8, targets=64),
        # The serving loop: a wave of 32 requests (16 shortest-path, 11 PPR, 5 label propagation).
        dict(name="serve-32-s18", kind="serve", graph="rmat", V=262144, ef=16, wmax=1000, pruned=False, n=32,
             host=True, alpha=0.15, rmax=1e-7, iterations=30),
    ]


# log2 of the vertices a drawn case of a kind may have
_SCALES = {"sssp": (10, 22), "ppr": (10, 20.5), "sssp_batch": (10, 21), "ppr_batch": (10, 20),
           "adsorption": (10, 21), "adjoint": (10, 19.5), "serve": (10, 17.5)}


def draw(rng):
    kind = rng.choice(["sssp", "sssp", "ppr", "ppr", "sssp_batch", "sssp_batch", "ppr_batch", "ppr_batch",
                       "adsorption", "adjoint", "serve"])
    lo, hi = _SCALES[kind]
    V = int(2 ** rng.uniform(lo, hi)) | rng.randrange(2)
    c = dict(kind=kind, graph=rng.choice(["rmat", "rmat", "uniform"]), V=V, ef=rng.randrange(5, 17),
             wmax=rng.choice([100, 1000]), pruned=False, n=1, host=rng.random() < 0.5)
    if kind in ("sssp_batch", "ppr_batch"):
        c["n"] = int(2 ** rng.uniform(1, 8.01))
    if kind == "serve":
        c["n"] = rng.randrange(8, 33)
    if kind in ("serve", "adjoint"):
        c["host"] = True
    if kind in ("sssp", "sssp_batch", "ppr_batch"):
        c["pruned"] = rng.random() < 0.3
    if c["host"]:  # a call whose results go to the host is kept below half a gigabyte of them
        c["n"] = max(1, min(c["n"], (1 << 27) // c["V"])) if kind.endswith("_batch") else c["n"]
    if kind in ("ppr", "ppr_batch", "adjoint", "serve"):
        c["alpha"] = rng.choice([0.15, 0.2])
        c["rmax"] = rng.choice([0.0, 1e-7]) if kind in ("ppr", "ppr_batch") else 1e-7
    if kind in ("adsorption", "serve"):
        c["iterations"] = 30 if kind == "serve" else rng.choice([10, 30])
    if kind == "adjoint":
        c["targets"] = rng.randrange(1, 129)
    return c


# ---- inputs ---------------------------------------------------------------------------


def _edges(case, seed):
    """The graph on the GPU, from the seed alone: (vlist, elist, wlist, flist), all sums in integers."""
    V, M = case["V"], case["V"] * case["ef"]
    want = M if case["kind"] == "adjoint" else 0
    if want:
        M = M * 8 // 5
    gen = torch.Generator("cuda")
    gen.manual_seed(1000003 * seed + V)
    if case["graph"] == "uniform":
        key = torch.randint(0, V * V, (M,), generator=gen, device="cuda")
        src, dst = key // V, key % V
    else:
        src = torch.zeros(M, dtype=torch.int64, device="cuda")
        dst = torch.zeros(M, dtype=torch.int64, device="cuda")
        for _ in range((V - 1).bit_length()):
            r = torch.rand(M, generator=gen, device="cuda")
            src.mul_(2).add_(r >= 0.76)
            dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        src.remainder_(V)
        dst.remainder_(V)
    key = torch.unique((src * V + dst)[src != dst])
    del src, dst
    if 0 < want < key.numel():
        key = key[torch.sort(torch.randperm(key.numel(), generator=gen, device="cuda")[:want])[0]]
    src, dst = key // V, key % V
    E = key.numel()
    del key
    row = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(torch.bincount(src, minlength=V), 0)
    w = torch.randint(1, case["wmax"] + 1, (E,), generator=gen, device="cuda", dtype=torch.int32)
    k = torch.randint(1, (1 << 20) + 1, (E,), generator=gen, device="cuda")
    total = torch.zeros(V, dtype=torch.int64, device="cuda").index_add_(0, src, k)
    f = (k.double() / total[src].double()).float()
    return row.int(), dst.int(), w, f


def _pick(row, n, seed):
    """n sources: half uniform over vertices with out-edges, half from the top 1% out-degree."""
    deg = np.diff(row)
    rng = np.random.default_rng(seed + 17)
    cand = np.flatnonzero(deg > 0)
    top = np.argsort(-deg, kind="stable")[:max(1, len(deg) // 100)]
    top = top[deg[top] > 0]
    half = n // 2
    return np.concatenate([rng.choice(cand, n - half), rng.choice(top, half)]).astype(np.int32)


def _pruned_dir(case, seed):
    """origin/ files of the graph in a new directory, pruned for the case's kind on the GPU."""
    d = tempfile.mkdtemp()
    os.mkdir(os.path.join(d, "origin"))
    for name, a in zip(("vlist", "elist", "wlist", "flist"), _edges(case, seed)):
        a.cpu().numpy().tofile(os.path.join(d, "origin", name + ".bin"))
    if case["kind"].startswith("sssp"):
        c2g.prune_sssp_device(d)
        return d, "sssp"
    c2g.prune_ppr_device(d, case["alpha"])
    return d, "ppr"


def _params(case, graph):
    p = graph.ppr_params(alpha=case["alpha"], pr0=case["alpha"], seeded=int(case["pruned"]), max_iter=500)
    if case["rmax"] > 0:
        p.rmax = case["rmax"]
    return p


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if case["pruned"]:
        d, variant = _pruned_dir(case, seed)
        try:
            row = np.fromfile(os.path.join(d, variant, "vlist.bin"), dtype=np.int32)
            g = c2g.Graph.load(d, variant)
        finally:
            shutil.rmtree(d)
    else:
        row, el, w, f = (a.cpu().numpy() for a in _edges(case, seed))
        need_w, need_f = kind.startswith("sssp") or kind == "serve", not kind.startswith("sssp")
        g = c2g.Graph.create(row, el, wlist=w if need_w else None, flist=f if need_f else None)
    torch.cuda.empty_cache()
    s = dict(case=case, graph=g, sources=_pick(row, n, seed))
    if kind in ("ppr", "ppr_batch", "adjoint"):
        s["params"] = _params(case, g)
    rng = np.random.default_rng(seed + 5)
    if kind in ("adsorption", "serve"):
        s["seeds"] = [rng.choice(g.V, 16, replace=False).astype(np.int32) for _ in range(max(1, n // 6))]
        s["p"] = rng.dirichlet((1.0, 1.0, 1.0), size=g.V).astype(np.float32).T.copy()
    if kind == "adjoint":
        s["targets"] = rng.choice(g.V, case["targets"], replace=False).astype(np.int32)
    if kind == "serve":
        s["server"] = c2g.Server(g, max_batch=64, alpha=case["alpha"], rmax=case["rmax"],
                                 ads_iterations=case["iterations"], p_inj=s["p"][0], p_cont=s["p"][1],
                                 p_abnd=s["p"][2])
    elif not case["host"]:
        shape = (n, g.V) if kind.endswith("_batch") else (g.V, 16) if kind == "adsorption" else (g.V,)
        dtype = torch.int32 if kind.startswith("sssp") else torch.float32
        s["out"] = torch.empty(shape, dtype=dtype, device="cuda")
        if kind.startswith("ppr"):
            s["res"] = torch.empty(shape, dtype=dtype, device="cuda")
        if kind == "adsorption":
            s["p"] = torch.from_numpy(s["p"]).cuda()
    return s


# ---- one pass -------------------------------------------------------------------------


def run(s):
    case, g, src = s["case"], s["graph"], s["sources"]
    kind, host = case["kind"], case["host"]
    out = None if host or kind == "serve" else s["out"].data_ptr()
    if kind == "sssp":
        dist, _ = g.sssp(int(src[0]), seeds=case["pruned"], mode=c2g.SEEDS_EXACT, out_ptr=out)
        return dist if host else s["out"]
    if kind == "sssp_batch":
        dist, _ = g.sssp_batch(src, seeds=case["pruned"], mode=c2g.SEEDS_EXACT, out_ptr=out)
        return dist if host else s["out"]
    if kind == "ppr":
        pr, res, _ = g.ppr(int(src[0]), s["params"], pr_ptr=out, res_ptr=None if host else s["res"].data_ptr())
        return [pr, res] if host else [s["out"], s["res"]]
    if kind == "ppr_batch":
        pr, res, _ = g.ppr_batch(src, s["params"], pr_ptr=out, res_ptr=None if host else s["res"].data_ptr())
        return [pr, res] if host else [s["out"], s["res"]]
    if kind == "adsorption":
        if host:
            return g.adsorption(s["seeds"][0], s["p"][0], s["p"][1], s["p"][2], iterations=case["iterations"])[0]
        g.adsorption_device(s["seeds"][0], *(p.data_ptr() for p in s["p"]), out, iterations=case["iterations"])
        return s["out"]
    if kind == "adjoint":
        grad, pi, lam, loss, _ = g.ppr_adjoint(int(src[0]), s["targets"], s["params"], rmax_backward=case["rmax"])
        return [grad, pi, lam, loss]
    return _wave(s)


def _split(n):
    """Requests of a wave: (SSSP, PPR, label propagation), about 50/35/15."""
    ads = max(1, n // 6)
    return n // 2, n - n // 2 - ads, ads


def _wave(s):
    """A wave of requests, submitted together in a mixed order, waited for one by one."""
    V, srv, src = s["graph"].V, s["server"], s["sources"]
    n_s, n_p, n_a = _split(len(src))
    dist = np.empty((n_s, V), np.int32)
    pr = np.empty((n_p, V), np.float32)
    labels = np.empty((n_a, V, 16), np.float32)
    tickets = []
    for i in range(max(n_s, n_p, n_a)):
        if i < n_s:
            tickets.append(srv.submit(c2g.REQ_SSSP, source=int(src[i]), out=dist[i]))
        if i < n_p:
            tickets.append(srv.submit(c2g.REQ_PPR, source=int(src[n_s + i]), out=pr[i]))
        if i < n_a:
            tickets.append(srv.submit(c2g.REQ_ADSORPTION, seeds=s["seeds"][i], out=labels[i]))
    for t in tickets:
        status, _ = srv.wait(t)
        if status != c2g.OK:
            raise RuntimeError("request failed with status %d" % status)
    return [dist, pr, labels]


# ---- what a pass cannot do without ------------------------------------------------------


def work(case):
    """Each input read once (row bounds, and target and weight of every edge), each result written once; the
    arithmetic of one pass over the edges (per label and iteration for the label propagation)."""
    V, E, n, kind = case["V"], case["V"] * case["ef"], case["n"], case["kind"]
    graph = 4.0 * V + 8.0 * E
    if kind.startswith("sssp"):
        return {"bytes": graph + 4.0 * V * n, "flops": 0.0}
    if kind.startswith("ppr"):
        return {"bytes": graph + 8.0 * V * n, "flops": 2.0 * E * n}
    if kind == "adsorption":
        return {"bytes": graph + 8.0 * V + 64.0 * V, "flops": 32.0 * E * case["iterations"]}
    if kind == "adjoint":
        return {"bytes": graph + 4.0 * E + 8.0 * V, "flops": 6.0 * E}
    n_s, n_p, n_a = _split(n)
    return {"bytes": graph + 4.0 * E + 4.0 * V * (n_s + n_p + 16 * n_a + 2),
            "flops": 2.0 * E * n_p + 32.0 * E * n_a * case["iterations"]}


# ---- the results in 64 bits --------------------------------------------------------------


def _pull_matrix(row, col, w):
    """P^T of the graph as a sparse matrix: row v holds the in-edges of v."""
    V = len(row) - 1
    src = torch.repeat_interleave(torch.arange(V, device="cuda"), torch.diff(row.long()))
    order = torch.argsort(col.long() * V + src)
    ptr = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(col.long(), minlength=V), 0)
    return torch.sparse_csr_tensor(ptr, src[order], w.double()[order], size=(V, V))


def _push(A, res, pr, active, alpha, rmax, absorb, max_iter):
    """Rounds of the push over the columns of res: active vertices send (1 - alpha) r w and keep nothing."""
    for _ in range(max_iter):
        if not bool(active.any()):
            break
        x = torch.where(active, res, 0.0).mul_(1.0 - alpha)
        res = torch.where(active, 0.0, res)
        del active
        res = res.add_(A @ x)
        active = res > rmax
        pr = pr.add_(torch.where(active, res, 0.0), alpha=absorb)
    return pr, res


def _ppr64(A, V, src, alpha, rmax, pr0, first=None):
    """(pr, res) of the sources, query-major; `first` gives a source's (vertices, weights) of the first hop."""
    prs, rs = [], []
    for at in range(0, len(src), 32):
        part = src[at:at + 32]
        pr = torch.zeros((V, len(part)), dtype=torch.float64, device="cuda")
        res = torch.zeros_like(pr)
        active = torch.zeros_like(pr, dtype=torch.bool)
        for q, v in enumerate(part):
            v = int(v)
            if first is None:
                pr[v, q], res[v, q], active[v, q] = pr0, 1.0, True
                continue
            pr[v, q] = alpha
            to, wt = first(v)
            pr[:, q].index_add_(0, to, wt * ((1.0 - alpha) * alpha))
            res[:, q].index_add_(0, to, wt * (1.0 - alpha))
            active[to, q] = True
        pr, res = _push(A, res, pr, active, alpha, rmax, alpha, 500)
        prs.append(pr.t().contiguous())
        rs.append(res.t().contiguous())
    return torch.cat(prs), torch.cat(rs)


def _labels64(A, V, seeds, p, iterations):
    inject = torch.zeros((V, 16), dtype=torch.float64, device="cuda")
    inject[torch.from_numpy(seeds).cuda().long(), torch.arange(16, device="cuda")] = 1.0
    p = torch.from_numpy(p).cuda().double()
    y = inject
    for _ in range(iterations):
        y = p[0][:, None] * inject + p[1][:, None] * (A @ y)
    return y


def exact(case, seed):
    kind, V = case["kind"], case["V"]
    if kind.startswith("sssp"):
        return None
    if case["pruned"]:
        d, variant = _pruned_dir(case, seed)
        try:
            names = ("vlist", "elist", "wlist", "hvlist", "helist", "hwlist")
            arrays = [torch.from_numpy(np.fromfile(os.path.join(d, variant, x + ".bin"),
                                                   dtype=np.float32 if x in ("wlist", "hwlist") else np.int32))
                      for x in names]
        finally:
            shutil.rmtree(d)
        row, col, f, hv, he, hw = (a.cuda() for a in arrays)
    else:
        row, col, _, f = _edges(case, seed)
    src = _pick(row.cpu().numpy(), case["n"], seed)
    A = _pull_matrix(row, col, f)
    rng = np.random.default_rng(seed + 5)
    if kind in ("adsorption", "serve"):
        seeds = [rng.choice(V, 16, replace=False).astype(np.int32) for _ in range(max(1, case["n"] // 6))]
        p = rng.dirichlet((1.0, 1.0, 1.0), size=V).astype(np.float32).T.copy()
        if kind == "adsorption":
            return _labels64(A, V, seeds[0], p, case["iterations"])
    alpha = float(np.float32(case["alpha"]))
    rmax = float(np.float32(case["rmax"]) if case["rmax"] > 0 else np.float32(0.001) / np.float32(V + 1))
    if kind == "serve":
        n_s, n_p, _ = _split(case["n"])
        labels = torch.stack([_labels64(A, V, x, p, case["iterations"]) for x in seeds])
        return [None, _ppr64(A, V, src[n_s:n_s + n_p], alpha, rmax, alpha)[0], labels]
    if kind == "adjoint":
        targets = rng.choice(V, case["targets"], replace=False)
        pi = _ppr64(A, V, src, alpha, rmax, alpha)[0][0]
        lam = torch.zeros((V, 1), dtype=torch.float64, device="cuda")
        lam[torch.from_numpy(targets).cuda()] = 1.0
        At = torch.sparse_csr_tensor(row.long(), col.long(), f.double(), size=(V, V))
        lam, _ = _push(At, lam.clone(), lam.clone(), lam > 0, alpha, rmax, 1.0, 500)
        lam = lam[:, 0]
        u = torch.repeat_interleave(torch.arange(V, device="cuda"), torch.diff(row.long()))
        return [(1.0 - alpha) * pi[u] * lam[col.long()], pi, lam, float(pi[torch.from_numpy(targets).cuda()].sum())]
    first = None
    if case["pruned"]:
        def first(v):
            a, b, c, e = int(hv[v]), int(hv[v + 1]), int(row[v]), int(row[v + 1])
            return torch.cat([he[a:b], col[c:e]]).long(), torch.cat([hw[a:b], f[c:e]]).double()
    pr, res = _ppr64(A, V, src, alpha, rmax, alpha, first)
    return [pr[0], res[0]] if kind == "ppr" else [pr, res]

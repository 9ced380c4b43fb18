"""The work that a user of this framework has it do, as measurable cases.

A user turns BOLD series into graphs and graphs into per-node metrics.  Two
scales are met in earnest: region graphs (90 to 1024 nodes, 1200 samples,
r > 0.2, weighted -- one call each, or hundreds of graphs in a batch) and
voxel graphs (thousands to 58,000 nodes, 120 to 240 samples, the top half to
two percent of the pairs, signed or absolute r, binary or weighted).  The
series are AR(1) noise with phi = 0.5 plus latent signals shared by the
voxels, the distribution of this repository's benchmark.

Every case goes through the public Python front end (or, where the result
stays on the device, the C entry point beneath it) and returns what the call
returns, whole.  One Context serves the process, as in a user's program.
"""
from __future__ import annotations

import ctypes as ct
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "pagani-toolkit_b200"))

import pagani  # noqa: E402

_CTX = None


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = pagani.Context(0)
    return _CTX


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: one atlas-sized weighted region graph from a host
        # series; launches and host round trips are what it costs
        dict(name="roi_build", kind="roi_build", N=90, T=1200, weighted=True, r=0.2),
        # the benchmark's subject: 58,000 voxels, top 1% of |r|, binary
        dict(name="voxel_build", kind="voxel_build", N=58000, T=240, sparsity=1.0, sign="abs", weighted=False,
             precision="bf16x3"),
        # a weighted voxel graph, odd sizes, signed r
        dict(name="voxel_build_weighted", kind="voxel_build", N=25211, T=187, sparsity=1.0, sign="signed",
             weighted=True, precision="bf16x3"),
        # the full correlation matrix of a 5,000-voxel subject for a .cormat file
        dict(name="correlation", kind="correlation", N=5000, T=200, weighted=False),
        # weighted path length and Onnela clustering of 512 region graphs in one call
        dict(name="fw_batch", kind="fw_batch", graphs=512, n_min=90, n_max=1024, T=1200, r=0.2),
        # weighted path length of one mid-sized graph
        dict(name="fw_single", kind="fw_single", N=2500, T=240, sparsity=5.0, dist=False),
        # per-node metrics of a weighted voxel graph: strength, Onnela
        # clustering, eigenvector centrality, participation coefficient
        dict(name="weighted_nodes", kind="weighted_nodes", N=25211, T=187, sparsity=1.0, modules=40),
        # per-node metrics of a binary voxel graph: degree, clustering, hop
        # path length and efficiency (the chain that every surrogate runs)
        dict(name="hop_metrics", kind="hop_metrics", N=40009, T=200, sparsity=0.5),
        # Brandes betweenness from all sources, with the hop path length
        dict(name="betweenness", kind="betweenness", N=30000, T=240, sparsity=1.0),
        # Newman leading-eigenvector modules
        dict(name="newman", kind="newman", N=16000, T=240, sparsity=1.0, weighted=False),
        # a whole 5,000-voxel subject in one call: build, every metric, Maslov
        # surrogates with their clustering and path length
        dict(name="subject", kind="subject", N=5000, T=200, r=0.3, surrogates=5, swaps=10),
        # subject-averaged Fisher-z graph of a small cohort
        dict(name="cohort", kind="cohort", N=16000, T=240, subjects=3, sparsity=1.0, fisher=True, weighted=True),
    ]


def _log_int(rng, lo, hi):
    """A size between lo and hi, even over its logarithm, mostly odd."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["roi_build", "voxel_build", "voxel_build", "correlation", "fw_batch", "fw_single",
                       "weighted_nodes", "hop_metrics", "betweenness", "newman", "subject", "cohort"])
    sparsity = round(math.exp(rng.uniform(math.log(0.5), math.log(2.0))), 3)
    if kind == "roi_build":
        return dict(kind=kind, N=_log_int(rng, 90, 1024), T=_log_int(rng, 100, 1200),
                    weighted=rng.random() < 0.7, r=round(rng.uniform(0.15, 0.4), 3))
    if kind == "voxel_build":
        weighted = rng.random() < 0.5
        precision = "fp32" if rng.random() < 0.25 else "bf16x3"
        return dict(kind=kind, N=_log_int(rng, 2000, 30000 if weighted or precision == "fp32" else 58000),
                    T=rng.randint(120, 240), sparsity=sparsity if not weighted else min(sparsity, 1.0),
                    sign=rng.choice(["abs", "signed"]), weighted=weighted, precision=precision)
    if kind == "correlation":
        return dict(kind=kind, N=_log_int(rng, 300, 5000), T=rng.randint(120, 240), weighted=rng.random() < 0.5)
    if kind == "fw_batch":
        return dict(kind=kind, graphs=_log_int(rng, 8, 512), n_min=90, n_max=_log_int(rng, 200, 1024),
                    T=_log_int(rng, 200, 1200), r=round(rng.uniform(0.2, 0.4), 3))
    if kind == "fw_single":
        return dict(kind=kind, N=_log_int(rng, 300, 2500), T=rng.randint(120, 240),
                    sparsity=round(rng.uniform(2.0, 10.0), 2), dist=rng.random() < 0.5)
    if kind == "weighted_nodes":
        return dict(kind=kind, N=_log_int(rng, 1000, 25000), T=rng.randint(120, 240), sparsity=min(sparsity, 1.0),
                    modules=rng.randint(2, 200))
    if kind == "hop_metrics":
        return dict(kind=kind, N=_log_int(rng, 1000, 40000), T=rng.randint(120, 240), sparsity=min(sparsity, 0.5))
    if kind == "betweenness":
        return dict(kind=kind, N=_log_int(rng, 1000, 30000), T=rng.randint(120, 240), sparsity=min(sparsity, 1.0))
    if kind == "newman":
        return dict(kind=kind, N=_log_int(rng, 1000, 16000), T=rng.randint(120, 240), sparsity=min(sparsity, 1.0),
                    weighted=rng.random() < 0.3)
    if kind == "subject":
        return dict(kind=kind, N=_log_int(rng, 500, 5000), T=rng.randint(150, 240), r=0.3,
                    surrogates=rng.randint(1, 5), swaps=rng.randint(2, 10))
    return dict(kind=kind, N=_log_int(rng, 1000, 16000), T=rng.randint(120, 240), subjects=rng.randint(2, 3),
                sparsity=min(sparsity, 1.0), fisher=rng.random() < 0.6, weighted=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _series(N, T, signals, seed, groups=None):
    """(T, N) float32 on the GPU: AR(1) noise (phi 0.5, 50 samples of burn-in)
    plus `signals` latent signals with N(0, 0.3^2) loadings.  groups: column
    offsets of graphs that each have signals of their own."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn((T + 50, N), device="cuda", generator=gen)
    for t in range(1, T + 50):
        x[t].add_(x[t - 1], alpha=0.5)
    x = x[50:].contiguous()
    if signals:
        L = torch.randn((signals, N), device="cuda", generator=gen) * 0.3
        groups = groups or [0, N]
        S = torch.randn((len(groups) - 1, T, signals), device="cuda", generator=gen)
        for g in range(len(groups) - 1):
            for f in range(signals):   # one rank-1 update at a time: the same bits on every run
                x[:, groups[g]:groups[g + 1]].addcmul_(S[g, :, f:f + 1], L[f:f + 1, groups[g]:groups[g + 1]])
    return x


def _signals(case):
    return 10 if case["kind"] in ("roi_build", "subject", "correlation", "fw_batch") else 20


def _bold(case, seed, subject=0):
    return _series(case["N"], case["T"], _signals(case), seed * 1009 + 31 * subject + 7)


def _batch_sizes(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return [int(n) for n in rng.integers(case["n_min"], case["n_max"] + 1, size=case["graphs"])]


def _batch_bold(case, seed):
    off = [0]
    for n in _batch_sizes(case, seed):
        off.append(off[-1] + n)
    return _series(off[-1], case["T"], _signals(case), seed * 1009 + 7, off), off


def _module_labels(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 5))
    return rng.integers(1, case["modules"] + 1, size=case["N"]).astype(np.float32)


def _graph_opts(case):
    """Threshold of the graph that a metric case works on."""
    weighted = case["kind"] in ("weighted_nodes", "fw_single", "fw_batch") or case.get("weighted", False)
    if "sparsity" in case:
        signed = weighted or case["kind"] == "cohort"    # subject averages rank signed r
        return dict(mode="s", value=case["sparsity"], sign=case.get("sign", "signed" if signed else "abs"),
                    weighted=weighted)
    return dict(mode="r", value=case["r"], sign="signed", weighted=weighted)


def _ptr(x):
    return (x.data_ptr(), tuple(x.shape))


def _csr_buffers(N, sparsity, weighted):
    nnz = 2 * pagani.sparsity_edges(N, sparsity)
    return dict(R=torch.empty(N + 1, dtype=torch.int32, device="cuda"),
                C=torch.empty(nnz, dtype=torch.int32, device="cuda"),
                V=torch.empty(nnz, dtype=torch.float32, device="cuda") if weighted else None)


def _csr_room(N, weighted):
    """Host buffers with room for every pair of a region graph."""
    return dict(R=np.zeros(N + 1, np.int32), C=np.zeros(N * (N - 1), np.int32),
                V=np.zeros(N * (N - 1), np.float32) if weighted else None)


def _csr_to(ctx, g, buf):
    """The CSR into the caller's buffers, host arrays or device tensors."""
    on_device = isinstance(buf["R"], torch.Tensor)
    p = [None if buf[k] is None else ct.c_void_p(buf[k].data_ptr() if on_device else buf[k].ctypes.data)
         for k in ("R", "C", "V")]
    ctx._check(pagani.lib().pg_graph_to_csr(ctx.h, g.h, p[0], p[1], p[2], int(on_device)))


def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    st = dict(case=case, ctx=ctx)
    if kind == "fw_batch":
        x, off = _batch_bold(case, seed)
        parts = [x[:, a:b].contiguous() for a, b in zip(off[:-1], off[1:])]
        torch.cuda.synchronize()
        st["graphs"] = [ctx.build_graph(None, **_graph_opts(case), device_ptr=_ptr(p))[0] for p in parts]
        room = case["graphs"] * case["n_max"]
        st["out"] = dict(eff=np.zeros(room, np.float32), lp=np.zeros(len(parts)), cp=np.zeros(room, np.float32),
                         cp_mean=np.zeros(len(parts)))
    elif kind == "cohort":
        st["bolds"] = [_bold(case, seed, s) for s in range(case["subjects"])]
        st["out"] = _csr_buffers(case["N"], case["sparsity"], case["weighted"])
    else:
        x = _bold(case, seed)
        torch.cuda.synchronize()
        if kind in ("roi_build", "correlation", "subject"):
            st["bold"] = x.cpu().numpy()      # these calls take the series from the host
            if kind == "roi_build":
                st["out"] = _csr_room(case["N"], case["weighted"])
        elif kind == "voxel_build":
            st["bold"] = x
            st["out"] = _csr_buffers(case["N"], case["sparsity"], case["weighted"])
        else:
            st["graph"] = ctx.build_graph(None, **_graph_opts(case), device_ptr=_ptr(x))[0]
        if kind == "weighted_nodes":
            st["modules"] = _module_labels(case, seed)
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------- the calls
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "roi_build":
        g, _ = ctx.build_graph(st["bold"], **_graph_opts(case))
        out = st["out"]
        _csr_to(ctx, g, out)
        g.free()
        return {k: v for k, v in out.items() if v is not None}
    if kind == "voxel_build":
        g, info = ctx.build_graph(None, **_graph_opts(case), precision=case["precision"],
                                  device_ptr=_ptr(st["bold"]))
        out = st["out"]
        _csr_to(ctx, g, out)
        g.free()
        res = dict(R=out["R"], C=out["C"], tau=info["tau"], edges=info["edges"])
        if out["V"] is not None:
            res["V"] = out["V"]
        return res
    if kind == "correlation":
        return ctx.correlation_packed(st["bold"], weighted=case["weighted"])
    if kind == "fw_batch":
        out = st["out"]
        p = {k: ct.c_void_p(v.ctypes.data) for k, v in out.items()}
        handles = (ct.c_void_p * len(st["graphs"]))(*[g.h.value for g in st["graphs"]])
        ctx._check(pagani.lib().pg_fw_batched(ctx.h, handles, len(handles), p["eff"], p["lp"], p["cp"],
                                              p["cp_mean"]))
        return out
    if kind == "fw_single":
        out = ctx.fw_paths(st["graph"], want_dist=case["dist"])
        return list(out)
    g = st.get("graph")
    if kind == "weighted_nodes":
        strength, isolated = ctx.degree(g)
        cp, _, cp_mean = ctx.clustering(g, kind="onnela")
        ec, lam, _, residual = ctx.eigen_centrality(g)
        pc, pcn, K = ctx.participation(g, st["modules"])
        return dict(strength=strength, isolated=isolated, cp=cp, cp_mean=cp_mean, ec=ec, eigenvalue=lam, pc=pc,
                    pc_norm=pcn, K=K)
    if kind == "hop_metrics":
        deg, isolated = ctx.degree(g)
        cp, tri, cp_mean = ctx.clustering(g)
        eff, inv, lp, hist, diameter = ctx.paths(g)
        return dict(deg=deg, isolated=isolated, cp=cp, tri=tri, cp_mean=cp_mean, eff=eff, inv=inv, lp=lp, hist=hist,
                    diameter=diameter)
    if kind == "betweenness":
        bc, bc64, eff, lp = ctx.betweenness(g, with_paths=True)
        return dict(bc=bc, bc64=bc64, eff=eff, lp=lp)
    if kind == "newman":
        labels, Q, modules = ctx.newman_weighted(g) if case["weighted"] else ctx.newman(g)
        return dict(labels=labels, Q=Q, modules=modules)
    if kind == "subject":
        return ctx.run_subjects([st["bold"]], mode="r", value=case["r"], sign="signed",
                                n_random=case["surrogates"], swaps_per_edge=case["swaps"])[0]
    # cohort
    with ctx.cohort(case["N"], fisher=case["fisher"], weighted=case["weighted"]) as c:
        for x in st["bolds"]:
            c.add(device_ptr=_ptr(x))
        g, info = c.graph(mode="s", value=case["sparsity"])
    out = st["out"]
    _csr_to(ctx, g, out)
    g.free()
    res = dict(R=out["R"], C=out["C"], tau=info["tau"], edges=info["edges"])
    if out["V"] is not None:
        res["V"] = out["V"]
    return res


# ----------------------------------------------------- bytes and operations
def work(case):
    """Bytes: the call's inputs once and its results once.  Operations: 2 per
    term of a correlation, 2 per min-plus update, one add per edge and source
    and sweep of a path computation, 2 per edge and step of a power method."""
    kind = case["kind"]
    if kind == "fw_batch":
        lo, hi = case["n_min"], case["n_max"]
        n1, n2, n3 = (lo + hi) / 2, (lo * lo + lo * hi + hi * hi) / 3, (lo + hi) * (lo * lo + hi * hi) / 4
        edges = 0.3 * n2
        return dict(bytes=case["graphs"] * (8 * edges + 8 * n1), flops=case["graphs"] * (2 * n3 + 0.3 * n2 * 2))
    N, T = case["N"], case["T"]
    M1 = N * (N - 1) // 2
    k = int(M1 * case["sparsity"] / 100) if "sparsity" in case else int(0.05 * M1)
    nnz = 2 * k
    if kind == "roi_build":
        return dict(bytes=4 * N * T + 4 * N + 0.3 * M1 * 2 * (8 if case["weighted"] else 4), flops=2 * T * M1)
    if kind == "voxel_build":
        return dict(bytes=4 * N * T + 4 * N + nnz * (8 if case["weighted"] else 4), flops=2 * T * M1)
    if kind == "correlation":
        return dict(bytes=4 * N * T + 4 * M1, flops=2 * T * M1)
    if kind == "fw_single":
        return dict(bytes=8 * nnz + 4 * N + (4 * N * N if case["dist"] else 0), flops=2 * N ** 3)
    if kind == "weighted_nodes":
        wedges = nnz * (nnz / N)
        return dict(bytes=8 * nnz + 32 * N, flops=wedges + 30 * 2 * nnz + 3 * nnz)
    if kind == "hop_metrics":
        return dict(bytes=4 * nnz + 36 * N, flops=nnz * (nnz / N) / 2 + 2 * nnz * N / 64)
    if kind == "betweenness":
        return dict(bytes=4 * nnz + 16 * N, flops=2 * nnz * N)
    if kind == "newman":
        return dict(bytes=4 * nnz + 4 * N, flops=2000 * 2 * nnz)
    if kind == "subject":
        per = 2 * nnz * N / 64
        return dict(bytes=4 * N * T + 24 * N + case["surrogates"] * 8 * nnz,
                    flops=2 * T * M1 + 2 * nnz * N + (1 + case["surrogates"]) * per)
    return dict(bytes=case["subjects"] * 4 * N * T + 4 * N + nnz * (8 if case["weighted"] else 4),
                flops=case["subjects"] * 2 * T * M1)


# ------------------------------------------------- the results in 64 bits
def _zscores(x):
    """(N, T) float64 rows of unit length; a constant voxel becomes zero."""
    z = x.double()
    z = z - z.mean(0)
    s = z.square().sum(0).sqrt()
    return torch.where(s > 0, z / s, torch.zeros_like(z)).t().contiguous()


def _fisher_mean(zs, fisher, i0, i1):
    acc = None
    for z in zs:
        r = z[i0:i1] @ z.t()
        r = torch.atanh(r) if fisher else r
        acc = r if acc is None else acc + r
    acc = acc / len(zs)
    return torch.tanh(acc) if fisher else acc


def _edges(case, zs):
    """Rows, columns (i < j) and 64-bit r of the graph's undirected edges."""
    o = _graph_opts(case)
    N = zs[0].shape[0]
    fisher = case.get("fisher", False)

    def keys(i0, i1):
        r = _fisher_mean(zs, fisher, i0, i1)
        return r.abs() if o["sign"] == "abs" else r

    cut, k = o["value"], None
    if o["mode"] == "s":
        k = pagani.sparsity_edges(N, o["value"])
        step = max(1, N // 64)
        samp = torch.cat([keys(i, i + 1)[0, i + 1:] for i in range(0, N, step)])
        q = min(0.999, 1.5 * k / (N * (N - 1) / 2) + 0.002)
        cut = torch.topk(samp, max(1, int(q * samp.numel()))).values[-1].item()
    ii, jj, rr = [], [], []
    for i0 in range(0, N, 1024):
        i1 = min(N, i0 + 1024)
        r = keys(i0, i1)
        m = r > cut
        m &= torch.arange(N, device="cuda")[None, :] > torch.arange(i0, i1, device="cuda")[:, None]
        i, j = m.nonzero(as_tuple=True)
        ii.append(i + i0)
        jj.append(j)
        rr.append(r[i, j])
    i, j, r = torch.cat(ii), torch.cat(jj), torch.cat(rr)
    if k is not None:
        r, top = torch.topk(r, k)
        i, j = i[top], j[top]
    return i, j, r


def _csr(N, i, j, r):
    row, col, val = torch.cat([i, j]), torch.cat([j, i]), torch.cat([r, r])
    order = torch.argsort(row * N + col)
    row, col, val = row[order], col[order], val[order]
    R = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    R[1:] = torch.cumsum(torch.bincount(row, minlength=N), 0)
    return R.to(torch.int32), row, col, val


def _dense(N, i, j, r=None, dtype=torch.float64):
    A = torch.zeros((N, N), dtype=dtype, device="cuda")
    v = torch.ones_like(i, dtype=dtype) if r is None else r.to(dtype)
    A[i, j] = v
    A[j, i] = v
    return A


def _host(x, dtype=None):
    return x.to(dtype).cpu().numpy() if dtype is not None else x.cpu().numpy()


def _shortest(W):
    """All-pairs min-plus closure of W (zero diagonal), 64 bits."""
    for k in range(W.shape[0]):
        torch.minimum(W, W[:, k:k + 1] + W[k:k + 1, :], out=W)
    return W


def _weighted_paths(i, j, w, n):
    W = _dense(n, i, j, 1.0 / w)
    W[W == 0] = math.inf
    W.fill_diagonal_(0.0)
    D = _shortest(W)
    x = torch.where((D >= 0.1) & ~torch.eye(n, dtype=torch.bool, device="cuda"), 1.0 / D, torch.zeros_like(D)).sum(1)
    eff = x / (n - 1)
    eff = torch.where(eff < 1.0 / n, torch.zeros_like(eff), eff)
    t = x.sum().item()
    return eff, (1.0 / (t / n / (n - 1)) if t > 0 else math.inf), D


def _onnela(i, j, w, n):
    A = _dense(n, i, j, (w / w.max()) ** (1.0 / 3.0))
    t = ((A @ A) * A).sum(1)
    k = (A > 0).sum(1).double()
    return torch.where(k >= 2, t / (k * (k - 1)).clamp(min=1), torch.zeros_like(t))


def _triangles(A):
    t = torch.empty(A.shape[0], dtype=torch.float64, device="cuda")
    for a in range(0, A.shape[0], 4096):
        t[a:a + 4096] = ((A[a:a + 4096] @ A) * A[a:a + 4096]).sum(1, dtype=torch.float64)
    return t / 2


def _binary_cp(A):
    t, k = _triangles(A), A.sum(1).double()
    return t, torch.where(k >= 2, 2 * t / (k * (k - 1)).clamp(min=1), torch.zeros_like(t))


def _hops(A, max_hop=64):
    """Sum of 1/d per node and ordered pairs per distance, by frontier products."""
    N = A.shape[0]
    inv = torch.zeros(N, dtype=torch.float64, device="cuda")
    hist = np.zeros(max_hop + 1, np.int64)
    diameter = 0
    for a in range(0, N, 8192):
        seen = torch.zeros((min(8192, N - a), N), dtype=torch.bool, device="cuda")
        seen[torch.arange(seen.shape[0]), a + torch.arange(seen.shape[0])] = True
        front, d = seen.clone(), 0
        while True:
            d += 1
            front = ((front.to(A.dtype) @ A) > 0) & ~seen
            c = front.sum(1)
            tot = int(c.sum().item())
            if not tot:
                break
            seen |= front
            inv[a:a + seen.shape[0]] += c.double() / d
            if d <= max_hop:
                hist[d] += tot
            diameter = max(diameter, d)
    return inv, hist, diameter


def _brandes(A):
    N = A.shape[0]
    bc = torch.zeros(N, dtype=torch.float64, device="cuda")
    inv = torch.zeros(N, dtype=torch.float64, device="cuda")
    for a in range(0, N, 4096):
        b = min(N, a + 4096)
        src = torch.arange(a, b, device="cuda")
        sigma = torch.zeros((b - a, N), dtype=torch.float64, device="cuda")
        sigma[torch.arange(b - a), src] = 1.0
        dist = torch.full((b - a, N), -1, dtype=torch.int16, device="cuda")
        dist[torch.arange(b - a), src] = 0
        d, front = 0, sigma.clone()
        while True:
            nxt = front @ A
            nxt[dist >= 0] = 0.0
            hit = nxt > 0
            if not bool(hit.any()):
                break
            d += 1
            dist[hit] = d
            sigma += nxt
            inv += hit.sum(0).double() / d
            front = nxt
        delta = torch.zeros_like(sigma)
        for lv in range(d, 0, -1):
            on = dist == lv
            bc += torch.where(on, delta, torch.zeros_like(delta)).sum(0)
            c = torch.where(on, (1.0 + delta) / sigma, torch.zeros_like(delta))
            up = (c @ A) * sigma
            delta = torch.where(dist == lv - 1, up, delta)
    return bc, inv


def _power_method(A):
    """The CUEC tools' iteration: start at the node ids, stop at 1e-6."""
    n = A.shape[0]
    u = torch.arange(n, dtype=torch.float64, device="cuda")
    lam = u.norm()
    for _ in range(10000):
        x = u / lam
        y = A @ x
        e1, e2 = (y - u).norm().item(), (y + u).norm().item()
        last, u, nrm = x, y, y.norm()
        if e1 <= 1e-6 or e2 <= 1e-6:
            break
        lam = nrm
    return last, lam.item()


def _participation(row, col, val, label, N, K):
    s = torch.zeros(N, dtype=torch.float64, device="cuda").index_add_(0, row, val)
    m = torch.zeros(N * K, dtype=torch.float64, device="cuda").index_add_(0, row * K + label[col] - 1, val)
    p = 1.0 - (m.view(N, K) / s.clamp(min=1e-300)[:, None]).square().sum(1)
    return torch.where(s > 0, p, torch.zeros_like(p))


def exact(case, seed):
    kind = case["kind"]
    if kind == "newman":
        return None
    torch.backends.cuda.matmul.allow_tf32 = False
    if kind == "fw_batch":
        x, off = _batch_bold(case, seed)
        count, room = len(off) - 1, case["graphs"] * case["n_max"]
        res = dict(eff=np.zeros(room), lp=np.zeros(count), cp=np.zeros(room), cp_mean=np.zeros(count))
        for q, (a, b) in enumerate(zip(off[:-1], off[1:])):
            i, j, r = _edges(case, [_zscores(x[:, a:b].contiguous())])
            w = r.float().double()          # the graph stores 32-bit weights
            eff, res["lp"][q], _ = _weighted_paths(i, j, w, b - a)
            cp = _onnela(i, j, w, b - a)
            res["eff"][a:b], res["cp"][a:b], res["cp_mean"][q] = _host(eff), _host(cp), cp.mean().item()
        return res
    N = case["N"]
    zs = [_zscores(_bold(case, seed, s)) for s in range(case.get("subjects", 1))]
    if kind == "correlation":
        r = zs[0] @ zs[0].t()
        i, j = torch.triu_indices(N, N, 1, device="cuda")
        return _host(r[i, j])
    i, j, r = _edges(case, zs)
    if kind in ("roi_build", "voxel_build", "cohort"):
        R, _, col, val = _csr(N, i, j, r)
        if kind == "roi_build":
            out = dict(R=_host(R), C=np.zeros(N * (N - 1), np.int32))
            out["C"][:col.numel()] = _host(col, torch.int32)
            if case["weighted"]:
                out["V"] = np.zeros(N * (N - 1))
                out["V"][:val.numel()] = _host(val)
            return out
        res = dict(R=R, C=col.to(torch.int32), tau=r.min().item(), edges=int(r.numel()))
        if case["weighted"]:
            res["V"] = val
        return res
    if kind == "fw_single":
        eff, lp, D = _weighted_paths(i, j, r.float().double(), N)
        return [_host(eff), lp, _host(D)] if case["dist"] else [_host(eff), lp]
    if kind == "weighted_nodes":
        w = r.float().double()
        _, row, col, val = _csr(N, i, j, w)
        strength = torch.zeros(N, dtype=torch.float64, device="cuda").index_add_(0, row, val)
        cp = _onnela(i, j, w, N)
        ec, lam = _power_method(_dense(N, i, j, w))
        label = torch.from_numpy(_module_labels(case, seed)).cuda().long()
        K = int(label.max().item())
        p = _participation(row, col, val, label, N, K)
        return dict(strength=_host(strength), isolated=int((torch.bincount(row, minlength=N) == 0).sum().item()),
                    cp=_host(cp), cp_mean=cp.mean().item(), ec=_host(ec), eigenvalue=lam, pc=_host(p),
                    pc_norm=_host(p / ((K - 1) / K) if K != 1 else p), K=K)
    if kind == "betweenness":
        if N > 20000:
            return None          # dense 64-bit Brandes takes too long
        bc, inv = _brandes(_dense(N, i, j))
        t = inv.sum().item()
        return dict(bc=_host(bc), bc64=_host(bc), eff=_host(inv / (N - 1)), lp=N * (N - 1) / t if t > 0 else 0.0)
    A = _dense(N, i, j, dtype=torch.float32)     # 0/1: products are whole numbers below 2^24
    deg = A.sum(1)
    tri, cp = _binary_cp(A)
    inv, hist, diameter = _hops(A)
    t = inv.sum().item()
    lp = N * (N - 1) / t if t > 0 else 0.0
    if kind == "hop_metrics":
        return dict(deg=_host(deg), isolated=int((deg == 0).sum().item()), cp=_host(cp), tri=_host(tri, torch.int64),
                    cp_mean=cp.mean().item(), eff=_host(inv / (N - 1)), inv=_host(inv), lp=lp, hist=hist,
                    diameter=diameter)
    # subject: what has a value without the surrogates' random streams
    bc, _ = _brandes(A.double())
    return dict(degree=_host(deg), cp=_host(cp), eff=_host(inv / (N - 1)), bc=_host(bc), modules=None,
                edges=int(r.numel()), tau=case["r"], cp_mean=cp.mean().item(), lp=lp, Q=None, n_modules=None,
                gamma=None, sigma=None, surrogate_graph_replays=None, **{"lambda": None})

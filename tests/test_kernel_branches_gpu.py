"""Branches of the kernels' dispatch rules, at the sizes where they change,
against the oracle or an FP64 restatement."""
import numpy as np
import pytest

from oracle import oracle as O
from pagani import synth
from tests import graphs as G

pytestmark = pytest.mark.gpu


# ------------------------------------------------------------------ Onnela
def _hub(n):
    """Node 0 connected to every other one, a ring and random chords among them."""
    rng = np.random.default_rng(n)
    edges = [(0, i) for i in range(1, n)] + [(i, i % (n - 1) + 1) for i in range(1, n)]
    edges += [tuple(rng.integers(1, n, 2)) for _ in range(4 * n)]
    return G.csr_from_edges(n, edges, [np.float32(x) for x in rng.uniform(0.1, 1.0, len(edges))])


@pytest.mark.parametrize("n", [3, 31, 33, 257, 1537, 1538, 2100])
def test_onnela_row_lengths(ctx, n):
    """Rows on both sides of the roots kept in shared memory (1536)."""
    R, C, V = _hub(n)
    cp, _, mean = ctx.clustering(ctx.graph(R, C, V), kind="onnela")
    cp_or, mean_or = O.onnela(R, C, V)
    # FP64 sums of non-negative terms, rounded to float once: half an ulp each side
    np.testing.assert_allclose(cp, cp_or, rtol=2.0 ** -23, atol=0)
    assert mean == pytest.approx(mean_or, rel=2.0 ** -23)


@pytest.mark.parametrize("change", ["negative", "zero", "all_zero", "infinite", "nan"])
def test_onnela_unusual_weights(ctx, change):
    """Weights that the product of cube roots does not cover take the general kernel."""
    R, C, V = G.random_weighted(120, 0.3, 5)
    rows = np.repeat(np.arange(120), np.diff(R))
    lo, hi = np.minimum(rows, C), np.maximum(rows, C)
    pick = (lo * 7 + hi * 13) % 11 == 0
    V = V.copy()
    if change == "all_zero":
        V[:] = 0
    else:
        V[pick] = {"negative": -V[pick], "zero": 0.0, "infinite": np.inf, "nan": np.nan}[change]
    cp, _, _ = ctx.clustering(ctx.graph(R, C, V), kind="onnela")
    with np.errstate(all="ignore"):
        A = np.zeros((120, 120))
        has = np.zeros((120, 120), bool)
        A[rows, C] = V / (np.nanmax(V) if change == "nan" else V.max())
        has[rows, C] = True
        want = np.zeros(120)
        for u in range(120):
            nb = np.nonzero(has[u])[0]
            k = len(nb)
            t = 0.0
            for x, j in enumerate(nb):
                for h in nb[x + 1:]:
                    if has[j, h] and A[j, h] != 0:
                        t += (A[j, h] * A[u, j] * A[u, h]) ** (1.0 / 3.0) if A[j, h] * A[u, j] * A[u, h] >= 0 \
                            else np.nan
            want[u] = 2.0 * t / k / (k - 1) if k >= 2 else 0.0
    np.testing.assert_allclose(cp, want.astype(np.float32), rtol=2.0 ** -22, atol=0, equal_nan=True)


def test_onnela_rows_out_of_order(ctx):
    """Rows whose columns do not ascend: j's scan takes any order, as before
    (u's own row is searched, so only rows without pairs above are shuffled)."""
    R = np.array([0, 3, 6, 9, 12], np.int32)          # K4
    C = np.array([1, 2, 3, 0, 2, 3, 0, 1, 3, 0, 1, 2], np.int32)
    V = np.array([.5, .6, .7, .5, .8, .9, .6, .8, 1., .7, .9, 1.], np.float32)
    want, _, _ = ctx.clustering(ctx.graph(R, C, V), kind="onnela")
    C2, V2 = C.copy(), V.copy()
    C2[9:12], V2[9:12] = [1, 0, 2], [.9, .7, 1.]      # node 3's row, swapped
    got, _, _ = ctx.clustering(ctx.graph(R, C2, V2), kind="onnela")
    np.testing.assert_allclose(got[:3], want[:3], rtol=2.0 ** -22)


# ------------------------------------------------------ network construction
@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("N,T", [(2, 1), (33, 3), (90, 4), (65, 15), (130, 16), (257, 63), (300, 65), (140, 1201),
                                 (2896, 67), (2897, 66)])
def test_weighted_build_sizes(ctx, N, T, precision):
    """Lengths around the 4- and 16-sample steps of the FP64 recheck and the
    64-sample chunks of the z-scores; both sides of the list-everything rule
    (2,896 nodes).  Edge set and weights equal the FP64 oracle's."""
    bold = synth.bold_series(N, T, 4, 100 + N + T)
    for sign in ("signed", "abs"):
        g, info = ctx.build_graph(bold, mode="r", value=0.3, sign=sign, weighted=True, precision=precision)
        R, C, V = g.to_csr()
        z, _ = O.zscore(bold)
        Ro, Co, Vo = O.graph_r(O.corr_packed(z, weighted=True), N, 0.3, abs_mode=sign == "abs", weighted=True)
        assert np.array_equal(R, Ro) and np.array_equal(C, Co) and np.array_equal(V, Vo)
        assert info["edges"] == len(C) // 2


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("N,value", [(31, 40.0), (128, 30.0), (129, 5.0), (255, 0.26), (257, 0.24), (900, 100.0),
                                     (1030, 0.3), (1030, 0.2)])
def test_adjacency_bits_and_pair_list(ctx, N, value, precision):
    """Both forms of the decided edges (bits from 0.26 % of the pairs on, a
    list below), at tile edges, up to the complete graph."""
    bold = synth.bold_series(N, 60, 4, 300 + N)
    z, _ = O.zscore(bold)
    r = O.corr_packed(z)
    for sign in ("signed", "abs"):
        g, _ = ctx.build_graph(bold, mode="s", value=value, sign=sign, precision=precision, guard=1e-3)
        R, C, _ = g.to_csr()
        Ro, Co, _, _ = O.graph_k(r, N, O.sparsity_k(N, value), abs_mode=sign == "abs")
        assert np.array_equal(R, Ro) and np.array_equal(C, Co)


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
def test_wide_band_flushes(ctx, precision):
    """A guard so wide that most pairs go through the FP64 band."""
    bold = synth.bold_series(700, 90, 4, 12)
    z, _ = O.zscore(bold)
    for guard, thr in ((0.5, 0.1), (0.2, 0.0)):
        g, info = ctx.build_graph(bold, mode="r", value=thr, precision=precision, guard=guard)
        R, C, _ = g.to_csr()
        Ro, Co, _ = O.graph_r(O.corr_packed(z), 700, thr)
        assert np.array_equal(R, Ro) and np.array_equal(C, Co)
        assert info["band_pairs"] > 100000


@pytest.fixture(scope="module")
def large():
    """9,000 voxels: 71 tile rows, beyond the size from which one sampled
    histogram replaces the full one (16 tiles per SM)."""
    bold = synth.bold_series(9000, 48, 6, 77)
    z, _ = O.zscore(bold)
    return bold, O.corr_packed(z, weighted=True)   # no r near +-1: both range rules agree


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
@pytest.mark.parametrize("mode,value,sign,weighted", [("s", 1.0, "abs", False), ("s", 0.1, "signed", False),
                                                      ("s", 0.5, "signed", True), ("r", 0.45, "abs", False),
                                                      ("r", 0.55, "signed", True)])
def test_one_full_gram_pass(ctx, large, mode, value, sign, weighted, precision):
    bold, r = large
    g, info = ctx.build_graph(bold, mode=mode, value=value, sign=sign, weighted=weighted, precision=precision)
    R, C, V = g.to_csr()
    if mode == "s":
        Ro, Co, Vo, tau = O.graph_k(r, 9000, O.sparsity_k(9000, value), abs_mode=sign == "abs", weighted=weighted)
        assert info["tau"] == tau
    else:
        Ro, Co, Vo = O.graph_r(r, 9000, value, abs_mode=sign == "abs", weighted=weighted)
    assert np.array_equal(R, Ro) and np.array_equal(C, Co)
    if weighted:
        assert np.array_equal(V, Vo)


@pytest.mark.parametrize("weighted", [False, True])
def test_sample_that_misses_the_edges(ctx, large, weighted):
    """Voxels 128..255 share one signal: their tile (linear index 71, not a
    multiple of 8) is not sampled and holds all of the wanted edges."""
    bold = large[0].copy()
    rng = np.random.default_rng(3)
    bold[:, 128:256] = rng.standard_normal((48, 1)) + 0.2 * rng.standard_normal((48, 128))
    z, _ = O.zscore(bold.astype(np.float32))
    r = O.corr_packed(z, weighted=True)
    g, info = ctx.build_graph(bold, mode="s", value=0.01, sign="signed", weighted=weighted)
    R, C, V = g.to_csr()
    Ro, Co, Vo, tau = O.graph_k(r, 9000, O.sparsity_k(9000, 0.01), weighted=weighted)
    assert info["tau"] == tau and np.array_equal(R, Ro) and np.array_equal(C, Co)
    if weighted:
        assert np.array_equal(V, Vo)


# ------------------------------------------------------- Floyd-Warshall batch
@pytest.mark.parametrize("sizes", [[1], [2, 63], [64], [65, 3, 130], [127, 128, 129, 190, 64, 1, 66],
                                   [257] * 3 + [70] * 90, [30 + 7 * q for q in range(60)]])
def test_fw_team_batches(ctx, sizes):
    """One team, several, and the most (a batch of many graphs), with sizes at
    the 64-wide block edges, against the dense FP32 closure and the oracle's
    clustering; the results come back in the caller's order."""
    gs, csr = [], []
    for q, n in enumerate(sizes):
        R, C, V = G.random_weighted(n, 0.15 if n > 20 else 0.6, 1000 + q)
        V = np.zeros(0, np.float32) if len(C) == 0 else V
        csr.append((R, C, V))
        gs.append(ctx.graph(R, C, V))
    out = ctx.fw_batched(gs)
    for (R, C, V), (eff, lp, cp, cpm) in zip(csr, out):
        n = len(R) - 1
        D = np.full((n, n), np.inf, np.float32)
        rows = np.repeat(np.arange(n), np.diff(R))
        D[rows, C] = np.float32(1.0) / V
        np.fill_diagonal(D, 0.0)
        D = O.fw_dense(D)
        E = np.zeros((n, n))
        ok = (D >= 0.1) & ~np.eye(n, dtype=bool)
        E[ok] = 1.0 / D[ok].astype(np.float64)
        want = E.sum(1) / max(n - 1, 1)
        want[want < 1.0 / n] = 0.0
        # distances: sums of at most ~10 FP32 terms in any order
        np.testing.assert_allclose(eff, want, rtol=1e-5)
        t = E.sum()
        assert lp == pytest.approx(n * (n - 1) / t, rel=1e-5) if t > 0 else np.isinf(lp)
        cp_or, m_or = O.onnela(R, C, V)
        np.testing.assert_allclose(cp, cp_or, rtol=2.0 ** -22)
        assert cpm == pytest.approx(m_or, rel=2.0 ** -22)


# ---------------------------------------------------------------- hop paths
@pytest.mark.parametrize("n", [1, 2, 64, 255, 257, 511, 513, 1030])
@pytest.mark.parametrize("kind", ["islands", "edgeless", "chain", "random"])
def test_hop_paths_batches(ctx, n, kind):
    """Batches of 256 and 512 sources with isolated sources, batches that have
    no edge at all between batches that do, and many levels."""
    rng = np.random.default_rng(n)
    if kind == "edgeless":
        edges = []
    elif kind == "chain":
        edges = [(i, i + 1) for i in range(n - 1) if i % 97]
    elif kind == "islands":       # nodes 256.. isolated but for a pair at the end
        m = min(n, 200)
        edges = [tuple(rng.integers(0, m, 2)) for _ in range(3 * m)] + ([(n - 2, n - 1)] if n > 1 else [])
    else:
        edges = [tuple(rng.integers(0, n, 2)) for _ in range(4 * n)]
    R, C, _ = G.csr_from_edges(n, edges)
    eff, inv, lp, hist, diam = ctx.paths(ctx.graph(R, C), max_hop=128)
    inv_or, hist_or, lp_or, d_or = O.bfs_paths(R, C, max_hop=128)
    assert np.array_equal(hist, hist_or) and diam == d_or
    if d_or <= 64:                # farther distances are added as they are found
        assert np.array_equal(inv, inv_or)
    np.testing.assert_allclose(inv, inv_or, rtol=1e-13)
    assert lp == pytest.approx(lp_or, rel=1e-12)


# ------------------------------------------------------------------- Newman
@pytest.mark.parametrize("n,deg", [(64, 6), (257, 12), (1000, 40), (1025, 60), (2047, 50), (2049, 90), (4200, 30)])
@pytest.mark.parametrize("weighted", [False, True])
def test_newman_team_sizes(ctx, n, deg, weighted):
    """Single CTAs, clusters that exchange y through shared memory (up to 2048
    rows) and through global memory, 256 and 512 threads, hubs that leave CTAs
    of a cluster without rows: labels of the sequential oracle."""
    rng = np.random.default_rng(n + deg)
    block = np.arange(n) * 5 // n
    edges = []
    for _ in range(n * deg // 2):
        a = int(rng.integers(n))
        b = int(rng.integers(n))
        if block[a] == block[b] or rng.random() < 0.08:
            edges.append((a, b))
    if n == 257:
        edges += [(0, i) for i in range(1, n)] + [(1, i) for i in range(2, n)]
    w = [np.float32(x) for x in rng.uniform(0.3, 1.0, len(edges))]
    R, C, V = G.csr_from_edges(n, edges, w)
    if weighted:
        labels, Q, nm = ctx.newman_weighted(ctx.graph(R, C, V))
        lo, Qo, nmo = O.newman_weighted(R, C, V)
    else:
        labels, Q, nm = ctx.newman(ctx.graph(R, C))
        lo, Qo, nmo, _ = O.newman(R, C)
    assert nm == nmo and np.array_equal(labels, lo)
    assert Q == pytest.approx(Qo, abs=1e-9)


# ------------------------------------------------------------ FP64 Gram blocks
@pytest.mark.parametrize("N,T", [(2, 1), (5, 3), (127, 15), (128, 16), (129, 17), (257, 33), (600, 64), (1000, 240)])
@pytest.mark.parametrize("weighted", [False, True])
def test_correlation_packed_blocks(ctx, N, T, weighted):
    """Edges of the 128-voxel blocks and of the 16- and 4-sample steps, with a
    flat voxel and a pair of duplicates: every float of the FP64 oracle."""
    bold = synth.bold_series(N, T, 3, 40 + N + T)
    if N > 4:
        bold[:, 1] = 2.0
        bold[:, 3] = bold[:, 0]
    r = ctx.correlation_packed(bold, weighted=weighted)
    z, _ = O.zscore(bold)
    assert np.array_equal(r, O.corr_packed(z, weighted=weighted).astype(np.float32))


@pytest.mark.parametrize("N", [2049, 3001])
def test_large_results_reach_the_host(ctx, N):
    """Results above 8 MB (staged by several threads), ends that divide no
    chunk, against a copy of the same data made on the device side."""
    import ctypes as ct

    import pagani
    import torch
    bold = synth.bold_series(N, 20, 3, N)
    r = ctx.correlation_packed(bold)
    z, _ = O.zscore(bold)
    assert r.nbytes > 8 << 20 and np.array_equal(r, O.corr_packed(z).astype(np.float32))
    g, _ = ctx.build_graph(bold, mode="r", value=-0.05, sign="signed", weighted=True)
    R, C, V = g.to_csr()
    assert C.nbytes > 8 << 20
    dev = [torch.empty(len(x), dtype=t, device="cuda") for x, t in ((R, torch.int32), (C, torch.int32),
                                                                   (V, torch.float32))]
    ctx._check(pagani.lib().pg_graph_to_csr(ctx.h, g.h, *[ct.c_void_p(d.data_ptr()) for d in dev], 1))
    for host, d in zip((R, C, V), dev):
        assert np.array_equal(host, d.cpu().numpy())


@pytest.mark.parametrize("K", [1, 31, 32, 33, 65])
def test_participation_module_counts(ctx, K):
    """Module counts around a warp, rows shorter and longer than 32 entries,
    isolated nodes: the oracle's floats."""
    R, C, V = G.random_weighted(150, 0.4, K)
    R2 = np.concatenate([R, [R[-1], R[-1]]]).astype(np.int32)      # two isolated nodes
    mod = (np.random.default_rng(K).integers(1, K + 1, 152)).astype(np.float32)
    mod[0] = K
    for v in (V, None):
        g = ctx.graph(R2, C, v)
        pc, pn, k = ctx.participation(g, mod)
        pc_or, pn_or, k_or = O.participation(R2, C, v, mod)
        assert k == k_or and np.array_equal(pc, pc_or) and np.array_equal(pn, pn_or)

"""Floyd-Warshall results to the last bit: the 64-wide in-place scheme, whose
FP32 sums associate in one fixed order, restated in numpy."""
import numpy as np
import pytest

from pagani import synth

pytestmark = pytest.mark.gpu
B = 64


def _closed(D):
    """Blocked closure of D (float32) with the diagonal block and the panels
    closed step by step in place."""
    D = D.copy()
    n = len(D)
    for a in range(0, n, B):
        k = slice(a, min(a + B, n))
        dg, w = D[k, k].copy(), min(a + B, n) - a
        for s in range(w):
            dg = np.minimum(dg, dg[:, s, None] + dg[s])
        row, col = D[k].copy(), D[:, k].copy()
        for s in range(w):
            row = np.minimum(row, dg[:, s, None] + row[s])
            col = np.minimum(col, col[:, s, None] + dg[s])
        row[:, k], col[k] = dg, dg
        rest = D.copy()
        for s in range(w):
            rest = np.minimum(rest, col[:, s, None] + row[s])
        D = rest
        D[k], D[:, k] = row, col
    return D


def _eff_lp(D):
    """Efficiency and path length with the sums' order: a node's terms over 32
    lanes and a shuffle tree, the graph's over its nodes."""
    n = len(D)
    ok = (D >= np.float32(0.1)) & ~np.eye(n, dtype=bool)
    E = np.zeros((n, (n + 31) // 32 * 32))
    E[:, :n][ok] = 1.0 / D[ok].astype(np.float64)
    acc = np.zeros((n, 32))
    for v in range(0, E.shape[1], 32):
        acc = acc + E[:, v:v + 32]
    lane = np.arange(32)
    for o in (16, 8, 4, 2, 1):
        acc = acc + acc[:, lane ^ o]
    rows = acc[:, 0]
    eff = (rows / (n - 1)).astype(np.float32)
    eff[eff < np.float32(1.0) / np.float32(n)] = 0
    t = 0.0
    for x in rows:
        t += float(x)
    return eff, (1.0 / (t / n / (n - 1)) if t > 0 else np.inf)


def _region_graph(n, r, seed, both_ways=True):
    x = synth.bold_series(n, 200, 6, seed).astype(np.float64)
    c = np.corrcoef(x.T).astype(np.float32)
    if not both_ways:    # another weight in each direction
        c = c * np.random.default_rng(seed).uniform(0.8, 1.0, (n, n)).astype(np.float32)
    np.fill_diagonal(c, 0)
    D = np.full((n, n), np.inf, np.float32)
    D[c > r] = np.float32(1) / c[c > r]
    np.fill_diagonal(D, 0)
    R = np.concatenate([[0], np.cumsum((c > r).sum(1))]).astype(np.int32)
    return (R, np.nonzero(c > r)[1].astype(np.int32), c[c > r]), D


@pytest.mark.parametrize("r", [0.2, 0.25, 0.3, 0.35])
def test_batch_distances_to_the_last_bit(ctx, r):
    sizes = [90, 333, 64, 65, 127, 128, 129, 200, 257, 400, 511]
    made = [_region_graph(n, r, 50 + q) for q, n in enumerate(sizes)]
    out = ctx.fw_batched([ctx.graph(*csr) for csr, _ in made])
    for (_, D), (eff, lp, _, _) in zip(made, out):
        eff_w, lp_w = _eff_lp(_closed(D))
        assert np.array_equal(eff, eff_w) and lp == lp_w


@pytest.mark.parametrize("n,r,both_ways", [(65, 0.3, True), (130, 0.3, True), (257, 0.33, False), (700, 0.35, True),
                                           (321, 0.25, False)])
def test_distances_to_the_last_bit(ctx, n, r, both_ways):
    csr, D = _region_graph(n, r, n, both_ways)
    g = ctx.graph(*csr)
    eff, lp, dist = ctx.fw_paths(g, want_dist=True)
    want = _closed(D)
    assert np.array_equal(dist.reshape(n, n), want)
    eff_w, lp_w = _eff_lp(want)
    assert np.array_equal(eff, eff_w) and lp == lp_w


def test_bundles_of_teams_to_the_last_bit(ctx):
    """So many graphs that teams of CTAs take them in bundles, and the same
    graphs a few at a time: sizes mixed so that bundles hold several."""
    made = [_region_graph(n, 0.3, n) for n in (60, 65, 90, 100, 128, 130, 190, 200)]
    gs = [ctx.graph(*csr) for csr, _ in made]
    pick = np.random.default_rng(1).integers(0, len(gs), 1600)
    out = ctx.fw_batched([gs[q] for q in pick])
    few = ctx.fw_batched(gs)
    want = [_eff_lp(_closed(D)) for _, D in made]
    for q, (eff, lp, cp, cpm) in zip(pick, out):
        assert np.array_equal(eff, want[q][0]) and lp == want[q][1]
        assert np.array_equal(cp, few[q][2]) and cpm == few[q][3]

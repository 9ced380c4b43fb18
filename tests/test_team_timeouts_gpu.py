"""Waits of CTA teams that run out, with no GPU fault: a test hook makes one CTA
of every team hold back, the others give up after a millisecond, the call
returns PG_ERR_TIMEOUT, and the same context then computes as before."""
import numpy as np
import pytest

import pagani
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _times_out(ctx, call):
    pagani.lib().pg_debug_stall_next_team(ctx.h, 1_000_000)
    with pytest.raises(pagani.PaganiError) as e:
        call()
    assert e.value.status == 6                      # PG_ERR_TIMEOUT


@pytest.mark.parametrize("sizes", [[300], [65] * 8, [200] * 40 + [70] * 60])
def test_fw_team_barrier(ctx, sizes):
    gs = [ctx.graph(*G.random_weighted(n, 0.2, 9 + q)) for q, n in enumerate(sizes)]
    before = ctx.fw_batched(gs)
    _times_out(ctx, lambda: ctx.fw_batched(gs))
    for a, b in zip(before, ctx.fw_batched(gs)):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_fw_paths_barrier(ctx):
    g = ctx.graph(*G.random_weighted(260, 0.2, 3))
    eff, lp = ctx.fw_paths(g)
    _times_out(ctx, lambda: ctx.fw_paths(g))
    eff2, lp2 = ctx.fw_paths(g)
    assert np.array_equal(eff, eff2) and lp == lp2


@pytest.mark.parametrize("n,deg", [(400, 20), (1000, 40), (2047, 50)])
@pytest.mark.parametrize("weighted", [False, True])
def test_newman_exchange(ctx, n, deg, weighted):
    """Clusters of 4 and 16 CTAs that exchange their vector through shared
    memory: every CTA leaves both passes, and its copies in flight are drained."""
    rng = np.random.default_rng(n)
    block = np.arange(n) * 4 // n
    edges = [(a, b) for a, b in rng.integers(0, n, (n * deg, 2)) if block[a] == block[b] or rng.random() < 0.08]
    R, C, V = G.csr_from_edges(n, edges, [np.float32(x) for x in rng.uniform(0.3, 1.0, len(edges))])
    g = ctx.graph(R, C, V) if weighted else ctx.graph(R, C)
    run = ctx.newman_weighted if weighted else ctx.newman
    labels, Q, nm = run(g)
    _times_out(ctx, lambda: run(g))
    labels2, Q2, nm2 = run(g)
    assert nm == nm2 and Q == Q2 and np.array_equal(labels, labels2)

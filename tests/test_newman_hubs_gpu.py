"""Clusters some of whose CTAs own no rows: a hub's row is heavier than a CTA's
share of the edges, and first rows are rounded down to even ones.  Such a team
must not exchange its vector through shared memory."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import graphs as G

pytestmark = pytest.mark.gpu
CTAS, MIN_EDGES, PUSH_ROWS = 16, 2048, 2048   # as newman.cu's team rule has them for small graphs


def _first(R, rank):
    """First row of a CTA: where its share of the edges begins, even."""
    n = len(R) - 1
    if rank >= CTAS:
        return n
    return 0 if rank <= 0 else int(np.searchsorted(R, int(R[n]) * rank // CTAS, side="left")) & ~1


def _hubs(n, hubs, seed):
    rng = np.random.default_rng(seed)
    block = np.arange(n) * 4 // n
    edges = [(int(a), int(b)) for a, b in rng.integers(0, n, (13 * n, 2)) if block[a] == block[b] or rng.random() < 0.05]
    edges += [(h, i) for h in hubs for i in range(n) if i != h]
    return G.csr_from_edges(n, edges, [np.float32(x) for x in rng.uniform(0.3, 1.0, len(edges))])


@pytest.mark.parametrize("n,hubs", [(2040, (0,)), (2047, (0, 1)), (2048, (801, 802, 803)), (2001, (1999, 2000))])
@pytest.mark.parametrize("weighted", [False, True])
def test_ctas_without_rows(ctx, n, hubs, weighted):
    R, C, V = _hubs(n, hubs, n)
    assert n <= PUSH_ROWS and len(C) > CTAS // 2 * MIN_EDGES           # sixteen CTAs, few enough rows to exchange
    rows = [_first(R, r + 1) - _first(R, r) for r in range(CTAS)]
    assert min(rows) == 0 and sum(rows) == n
    if weighted:
        labels, Q, nm = ctx.newman_weighted(ctx.graph(R, C, V))
        lo, Qo, nmo = O.newman_weighted(R, C, V)
    else:
        labels, Q, nm = ctx.newman(ctx.graph(R, C))
        lo, Qo, nmo, _ = O.newman(R, C)
    assert nm == nmo and np.array_equal(labels, lo)
    assert Q == pytest.approx(Qo, abs=1e-9)

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

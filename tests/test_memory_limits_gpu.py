"""Calls in little device memory (a limit on the context's workspace stands in
for a full device): routes that want room to spare give way to those that do
not, and scratch of one call does not stay in the way of the next."""
import numpy as np
import pytest

import pagani
from pagani import synth
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _limit(c, bytes_):
    pagani.lib().pg_debug_memory_limit(c.h, int(bytes_))


# limits: what a build with exactly sized lists needs, with a tenth to spare
@pytest.mark.parametrize("N,T,mb,kw", [
    (2000, 100, 6, dict(mode="r", value=0.6)), (2000, 100, 6, dict(mode="r", value=0.6, weighted=True)),
    (2000, 100, 6, dict(mode="s", value=1.0)), (9000, 48, 10.5, dict(mode="r", value=0.6, weighted=True)),
    (9000, 48, 10.5, dict(mode="s", value=0.05)), (9000, 48, 30.5, dict(mode="s", value=1.0, precision="fp32"))])
def test_build_with_exact_lists(ctx, N, T, mb, kw):
    bold = synth.bold_series(N, T, 6, N)
    g, info = ctx.build_graph(bold, **kw)
    R, C, V = g.to_csr()
    with pagani.Context(0) as c:
        _limit(c, mb * 1e6)
        g2, info2 = c.build_graph(bold, **kw)
        R2, C2, V2 = g2.to_csr()
        assert np.array_equal(R, R2) and np.array_equal(C, C2) and info["tau"] == info2["tau"]
        assert np.array_equal(V, V2) if V is not None else V2 is None
        with pagani.Context(0) as none:      # and an error, not a crash, where nothing fits
            _limit(none, 1e6)
            with pytest.raises(pagani.PaganiError) as e:
                none.build_graph(bold, **kw)
            assert e.value.status == 3
        del g2


def test_scratch_of_a_build_makes_room(ctx):
    bold = synth.bold_series(9000, 48, 6, 9000)
    fw = G.random_weighted(2500, 0.01, 1)
    want = ctx.fw_paths(ctx.graph(*fw))
    with pagani.Context(0) as c:
        _limit(c, 60e6)                       # the build holds 46 MB, the sweep wants 30 more
        g, _ = c.build_graph(bold, mode="s", value=6.0)
        h = c.graph(*fw)
        eff, lp = c.fw_paths(h)
        assert np.array_equal(eff, want[0]) and lp == want[1]
        del g, h


def test_roots_of_onnela_make_room(ctx):
    R, C, V = G.random_weighted(3000, 0.25, 2)         # 2.2 million entries: 18 MB of roots
    want = ctx.clustering(ctx.graph(R, C, V), kind="onnela")[0]
    fw = G.random_weighted(1200, 0.02, 3)
    lp = ctx.fw_paths(ctx.graph(*fw))[1]
    with pagani.Context(0) as c:
        g, h = c.graph(R, C, V), c.graph(*fw)
        _limit(c, 22e6)
        assert np.array_equal(c.clustering(g, kind="onnela")[0], want)
        assert c.fw_paths(h)[1] == lp
        _limit(c, 2e6)                        # no room for roots: the kernel that needs none
        with pagani.Context(0) as d:
            _limit(d, 2e6)
            k = d.graph(R, C, V)
            np.testing.assert_allclose(d.clustering(k, kind="onnela")[0], want, rtol=2.0 ** -22)
            del k
        del g, h


def test_subject_that_could_not_be_added_does_not_count(ctx):
    """The largest limit at which an add still fails: all but its last buffer."""
    bolds = [synth.bold_series(260, 40, 4, s) for s in (1, 2)]

    def add(limit):
        with pagani.Context(0) as c, c.cohort(260, fisher=True) as avg:
            _limit(c, limit)
            try:
                avg.add(bolds[0])
                ok = True
            except pagani.PaganiError as e:
                assert e.status == 3
                ok = False
            assert avg.subjects == int(ok)
            _limit(c, 0)
            avg.add(bolds[1])
            return ok, avg.packed()
    with ctx.cohort(260, fisher=True) as alone:
        alone.add(bolds[1])
        want = alone.packed()
    lo, hi = 1 << 10, 1 << 24
    while hi - lo > 1:
        mid = (lo + hi) // 2
        ok, packed = add(mid)
        if ok:
            hi = mid
        else:
            lo = mid
            assert np.array_equal(packed, want)

"""Which FP64 solver KWG_SOLVER_AUTO takes at theta = 1/2: many PDEs of few nodes and few steps on ragged
uniform grids stream, all else runs on chip, in the uniform and the uneven call alike.  The routes are
told apart by their bits: streaming lanes and on-chip PDEs do not depend on their neighbours."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def prices(ctx, o, **kw):
    import kwg

    rc, p, st = ctx.fd1d_price(o, kwg.params(**kw))
    assert rc == kwg.KWG_OK, ctx.last_error()
    return p


@pytest.mark.parametrize("n,x_dim,t_dim,density,streams", [
    (16384, 32, 200, math.inf, False), (16384, 16, 200, math.inf, True), (8000, 16, 60, math.inf, False),
    (40000, 65, 3, math.inf, True), (40000, 65, 60, 0.25, False), (24000, 129, 3, math.inf, True),
    (24000, 128, 3, math.inf, False)])
def test_auto_takes_the_faster_solver(built, n, x_dim, t_dim, density, streams):
    import kwg
    import portfolio

    c = kwg.Context(0)  # no tuning record
    try:
        o = portfolio.american_portfolio(n, seed=x_dim)
        kw = dict(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=density)
        p, stream, chip = (prices(c, o, solver=s, **kw) for s in (kwg.SOLVER_AUTO, kwg.SOLVER_THOMAS, kwg.SOLVER_PCR))
        assert not np.array_equal(stream, chip, equal_nan=True)
        assert np.array_equal(p, stream if streams else chip, equal_nan=True)
        ok = np.isfinite(stream)
        assert np.all(np.abs(stream - chip)[ok] <= np.maximum(1e-10 * np.abs(stream), 1e-13 * o["k"])[ok])
    finally:
        c.close()


@pytest.mark.parametrize("n,nodes,levels,streams", [(30000, (8, 17), (10, 30), True), (30000, (90, 129), (30, 60), False),
                                                    (200, (8, 17), (10, 30), False)])
def test_uneven_auto_takes_the_faster_solver(built, n, nodes, levels, streams):
    import kwg
    import portfolio

    c = kwg.Context(0)
    try:
        rng = np.random.default_rng(n)
        o = portfolio.american_portfolio(n, seed=3)
        x, t = (rng.integers(*r, n).astype(np.int32) for r in (nodes, levels))
        got = {}
        for s in (kwg.SOLVER_AUTO, kwg.SOLVER_THOMAS, kwg.SOLVER_PCR):
            rc, got[s], _ = c.fd1d_price_uneven(o, x, t, kwg.params(scale=5.0, density=math.inf, solver=s))
            assert rc == kwg.KWG_OK, c.last_error()
        assert not np.array_equal(got[1], got[2], equal_nan=True)
        assert np.array_equal(got[0], got[1] if streams else got[2], equal_nan=True)
    finally:
        c.close()

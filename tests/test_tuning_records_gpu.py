"""The autotuner's records: which calls they bind."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(c, o, **kw):
    import kwg

    rc, p, st = c.fd1d_price(o, kwg.params(**kw))
    assert rc == kwg.KWG_OK, c.last_error()
    return p


def test_a_record_binds_its_own_scheme_and_kind_of_grid(built):
    """Tuned at theta = 1/2 on a uniform grid: calls of the same size with another theta, or on a sinh grid, run as
    in a context without records (told apart by their bits: another solver, another number of warps)."""
    import kwg
    import portfolio

    tuned, fresh = kwg.Context(0), kwg.Context(0)
    try:
        kw = dict(t_dim=40, x_dim=128, scale=5.0)
        o = portfolio.american_portfolio(9000, seed=2)
        rec = tuned.autotune_ex(kwg.params(density=math.inf, **kw), len(o))
        assert rec.solver == kwg.SOLVER_PCR  # 5 times the streaming solver's speed there
        for density in (math.inf, 0.25):
            assert np.array_equal(run(tuned, o, theta=0.6, density=density, **kw), run(fresh, o, theta=0.6, density=density, **kw))
        kw = dict(t_dim=200, x_dim=1024, scale=5.0, precision=kwg.FP32)
        o = portfolio.american_portfolio(6000, seed=3)
        rec = tuned.autotune_ex(kwg.params(density=math.inf, **kw), len(o))
        assert rec.option_warps == 1  # two on sinh grids
        assert np.array_equal(run(tuned, o, density=0.25, **kw), run(fresh, o, density=0.25, **kw))
    finally:
        tuned.close()
        fresh.close()


def test_an_uneven_record_binds_its_own_scheme(built):
    import kwg
    import portfolio

    tuned, fresh = kwg.Context(0), kwg.Context(0)
    try:
        o, x, t = portfolio.uneven_portfolio(600, seed=9)
        x, t = np.minimum(x, 300), np.minimum(t, 60)
        rec = tuned.autotune_uneven(o, x, t, kwg.params(scale=5.0, density=math.inf))
        assert rec.solver == kwg.SOLVER_PCR
        got = []
        for c in (tuned, fresh):
            rc, p, _ = c.fd1d_price_uneven(o, x, t, kwg.params(scale=5.0, density=math.inf, theta=0.7))
            assert rc == kwg.KWG_OK, c.last_error()
            got.append(p)
        assert np.array_equal(got[0], got[1], equal_nan=True)
    finally:
        tuned.close()
        fresh.close()


@pytest.mark.parametrize("x_dim,same", [(100, [0, 1, 2, 3]), (256, [2, 3]), (1500, [0, 1]), (1500, [2, 3])])
def test_fp32_choices_that_run_alike_share_one_time(built, x_dim, same):
    """Up to 128 nodes one warp, at least two above 1024, never more than four."""
    import kwg

    c = kwg.Context(0)
    try:
        t = c.autotune_ex(kwg.params(t_dim=30, x_dim=x_dim, scale=5.0, density=math.inf, precision=kwg.FP32), 300)
        ms = [*t.fp32_ms, t.fp32_8w_ms]
        assert min(ms) > 0 and len({ms[i] for i in same}) == 1
        assert ms[(1, 2, 4, 8).index(t.option_warps)] == min(ms) and t.option_warps != 8
    finally:
        c.close()

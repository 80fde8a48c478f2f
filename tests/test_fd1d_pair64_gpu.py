"""The on-chip solvers.  FP64 on FP32 units (what KWG_SOLVER_AUTO takes for theta = 1/2 and up to 2048
nodes): edges of its lane and warp layouts, the warps-per-PDE rule, and the PDEs it leaves
to the FP64 kernel.  Prices within 1e-10 relative of the oracle (or of the streaming FP64
solver), 1e-13 K absolute below 1e-3, as the library's other FP64 paths."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL, ABS_TOL = 1e-10, 1e-13


def mixed(n, seed):
    """American and European, puts and calls."""
    import portfolio

    o = portfolio.american_portfolio(n, seed=seed)
    o["e"] = np.arange(n) // 2 % 3 != 0
    return o


def check(got, want, k):
    assert np.isfinite(got).all()
    assert np.max(np.abs(got - want) / np.maximum(REL_TOL * np.abs(want), ABS_TOL * k)) <= 1.0


@pytest.mark.parametrize("density", [0.25, math.inf], ids=["sinh", "uniform"])
@pytest.mark.parametrize("x_dim", [3, 5, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 500, 512, 513, 1000, 1023, 1024,
                                   1025, 1500, 2047, 2048])
def test_grid_sizes(ctx, x_dim, density):
    """Every nodes-per-lane count, full and ragged lanes, the shortest grids."""
    import kwg
    import kwor

    o = mixed(24, seed=x_dim)
    kw = dict(t_dim=37, x_dim=x_dim, scale=5.0, density=density)
    rc, p, st = ctx.fd1d_price(o, kwg.params(**kw))
    assert rc == 0 and (st == 0).all(), ctx.last_error()
    rc, msg, want, _ = kwor.fd1d_price(o, **kw)
    assert rc == 0, msg
    check(p, want, o["k"])


@pytest.mark.parametrize("x_dim,density", [(200, 0.25), (512, math.inf), (500, 0.25), (1024, math.inf), (1024, 0.25)])
@pytest.mark.parametrize("n", [1, 152, 153, 304, 305, 700])
def test_warps_per_pde(ctx, n, x_dim, density):
    """PDE counts on both sides of the rule's lines (four, two and one warp per scheduler of
    152 SMs) against the streaming solver."""
    import kwg

    o = mixed(n, seed=n)
    kw = dict(t_dim=50, x_dim=x_dim, scale=5.0, density=density)
    rc, p, st = ctx.fd1d_price(o, kwg.params(**kw))
    assert rc == 0 and (st == 0).all()
    rc, want, _ = ctx.fd1d_price(o, kwg.params(solver=kwg.SOLVER_THOMAS, **kw))
    assert rc == 0
    check(p, want, o["k"])


def left_over(n):
    """Options whose PDEs FP32 cannot hold (a drift across the grid; calls on a grid that
    reaches e^90 and more; a degenerate factorisation) among ordinary ones."""
    o = mixed(n, seed=8)
    o["z"][3::7], o["r"][3::7], o["q"][3::7], o["t"][3::7] = 0.02, 0.2, 0.0, 5.0
    o["z"][5::11], o["t"][5::11], o["w"][5::11] = 1.5, 3.0, 1
    o["z"][6] = 1e200
    o["t"][9] = -1.0
    return o


@pytest.mark.parametrize("x_dim,scale,density", [(128, 5.0, math.inf), (300, 50.0, 0.25), (1100, 50.0, 0.25)])
@pytest.mark.parametrize("entry", ["host", "uneven"])
def test_left_over_pdes_take_the_fp64_kernel(ctx, entry, x_dim, scale, density):
    """Statuses and prices as the streaming solver's."""
    import kwg

    o = left_over(66)
    kw = dict(t_dim=60, x_dim=x_dim, scale=scale, density=density)
    rc, want, wst = ctx.fd1d_price(o, kwg.params(solver=kwg.SOLVER_THOMAS, **kw))
    assert rc == 0 and wst[6] == kwg.STATUS_SOLVER and wst[9] == kwg.STATUS_BAD_INPUT
    if entry == "host":
        rc, p, st = ctx.fd1d_price(o, kwg.params(**kw))
    else:
        rc, p, st = ctx.fd1d_price_uneven(o, np.full(len(o), x_dim), np.full(len(o), 60), kwg.params(scale=scale,
                                                                                                  density=density))
    assert rc == 0 and np.array_equal(st, wst)
    ok = st == 0
    assert ok.sum() > 0.5 * len(o)
    check(p[ok], want[ok], o["k"][ok])


def test_other_schemes_after_tuning(built):
    """A record made at theta = 1/2 on a grid beyond the FP64 on-chip kernel does not reach
    a call with another theta; small grids with many PDEs take the streaming solver."""
    import kwg
    import kwor

    c = kwg.Context(0)
    try:
        kw = dict(t_dim=24, x_dim=1500, scale=5.0, density=0.25)
        t = c.autotune_ex(kwg.params(**kw), 16)
        assert t.pcr_ms < 0
        o = mixed(16, seed=5)
        for theta in (0.5, 0.6):
            rc, p, st = c.fd1d_price(o, kwg.params(theta=theta, **kw))
            assert rc == 0 and (st == 0).all(), c.last_error()
            rc, msg, want, _ = kwor.fd1d_price(o, theta=theta, **kw)
            check(p, want, o["k"])
        many = mixed(8000, seed=6)
        kw = dict(t_dim=12, x_dim=18, scale=5.0, density=0.25)
        rc, p, st = c.fd1d_price(many, kwg.params(**kw))
        rc, want, wst = c.fd1d_price(many, kwg.params(solver=kwg.SOLVER_THOMAS, **kw))
        assert np.array_equal(p, want) and np.array_equal(st, wst)
    finally:
        c.close()


@pytest.mark.parametrize("theta", [0.5, 0.8])
@pytest.mark.parametrize("n,x_dim,density", [(1, 512, 0.25), (305, 512, 0.25), (700, 500, math.inf), (152, 1024, math.inf),
                                             (153, 1024, 0.25), (40, 2048, math.inf), (40, 2047, 0.25), (3, 3, 0.25),
                                             (9, 65, math.inf)])
def test_fp32_warps_per_pde(ctx, n, x_dim, density, theta):
    """FP32 stepping with the warp count left to the rule, against the streaming FP64 solver
    within the FP32 path's 1e-5 (a relative 2e-7 on the 3-node grid, whose prices are large)."""
    import kwg

    o = mixed(n, seed=n)
    kw = dict(t_dim=50, x_dim=x_dim, scale=5.0, density=density, theta=theta)
    rc, p, st = ctx.fd1d_price(o, kwg.params(precision=kwg.FP32, **kw))
    assert rc == 0 and (st == 0).all()
    rc, want, _ = ctx.fd1d_price(o, kwg.params(solver=kwg.SOLVER_THOMAS, **kw))
    assert rc == 0
    assert np.max(np.abs(p - want) - 2e-7 * np.abs(want)) <= 1e-5

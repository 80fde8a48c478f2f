"""FP64 precision of KWG_SOLVER_AUTO at theta = 1/2 on steep grids (large alpha = sigma^2 dt / 2 dx^2), FD1D and
its FD1D-BS control variate, against the scheme stepped in 64-bit increments here."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fd64(o, x_dim, t_dim, scale, density):
    """(1 - dt A / 2) d = dt A V, V += d, floored at the payoff: the increments carry 64 bits of
    their own, so the rounding left is V's.  The grid in extended precision."""
    N = x_dim
    t, z, r, q = (o[f].astype(np.longdouble) for f in ("t", "z", "r", "q"))
    half = scale * z * np.sqrt(t)
    y = (2 * np.arange(N, dtype=np.longdouble) / (N - 1) - 1)[:, None]
    x = half * y if math.isinf(density) else density * np.sinh(np.arcsinh(half / density) * y)
    dt, axx = t / (t_dim - 1), z * z / 2
    ax = r - q - axx
    up, span = x[1:] - x[:-1], x[2:] - x[:-2]
    al, be = np.zeros_like(x), np.zeros_like(x)
    al[1:-1] = dt * (2 * axx / up[1:] + ax) / span
    be[1:-1] = dt * (2 * axx / up[:-1] - ax) / span
    al[0], be[-1] = dt * ax / up[0], -dt * ax / up[-1]
    ga, al, be = (-r * dt).astype(float), al.astype(float), be.astype(float)
    p = np.maximum(0, np.where(o["w"] < 0, -1, 1) * np.expm1(x)).astype(float)
    floor = np.where(o["e"] != 0, p, -np.inf)
    floor[-1] = -np.inf
    b = 1 - 0.5 * (ga - al - be)
    m, c, ib = np.zeros_like(b), np.zeros_like(b), np.empty_like(b)
    ib[0] = 1 / b[0]
    for j in range(1, N):
        m[j] = -0.5 * be[j] * ib[j - 1]
        ib[j] = 1 / (b[j] + 0.5 * m[j] * al[j - 1])
    c[:-1] = -0.5 * al[:-1] * ib[:-1]
    V = p.copy()
    for _ in range(t_dim - 1):
        D = V[1:] - V[:-1]
        d = ga * V
        d[:-1] += al[:-1] * D
        d[1:] -= be[1:] * D
        for j in range(1, N):
            d[j] -= m[j] * d[j - 1]
        d *= ib
        for j in range(N - 2, -1, -1):
            d[j] -= c[j] * d[j + 1]
        V = np.maximum(V + d, floor)
    xs = np.log(o["s"] / o["k"])
    i = np.arange(len(o))
    hi = np.array([np.searchsorted(x[:, k].astype(float), xs[k]) for k in i])
    x0, x1 = x[hi - 1, i].astype(float), x[hi, i].astype(float)
    return o["k"] * ((x1 - xs) * V[hi - 1, i] + (xs - x0) * V[hi, i]) / (x1 - x0)


def european(o):
    t, z, r, q, s, k, w = (o[f].astype(float) for f in ("t", "z", "r", "q", "s", "k", "w"))
    zt = z * np.sqrt(t)
    d1 = (np.log(s / k) + (r - q + 0.5 * z * z) * t) / zt
    cdf = np.vectorize(lambda v: 0.5 * math.erfc(-v / math.sqrt(2.0)))
    return w * (s * cdf(w * d1) * np.exp(-q * t) - k * cdf(w * (d1 - zt)) * np.exp(-r * t))


@pytest.mark.parametrize("bs", [False, True], ids=["fd", "bs"])
@pytest.mark.parametrize("n,x_dim,scale,density", [(24, 512, 50.0, 0.25), (24, 1000, 5.0, 0.25), (24, 2048, 5.0, 0.25),
                                                   (500, 1024, 5.0, 0.25), (24, 512, 5.0, math.inf)])
def test_steep_grids(ctx, n, x_dim, scale, density, bs):
    """No further off than FP64 stepping (KWG_SOLVER_THOMAS), as far as the state's own rounding can be
    told: a pair of floats (2^-49 of the value), rounded about three times a step; over 39 steps, as independent
    errors, 3 sqrt(39) 2^-49 = 3.3e-14 of the price, for each of the control variate's two solves."""
    import kwg
    import portfolio

    t_dim = 40
    o = portfolio.american_portfolio(n, seed=x_dim + n)
    price = ctx.fd1d_bs_price if bs else ctx.fd1d_price
    want = fd64(o[:24], x_dim, t_dim, scale, density)
    if bs:
        euro = o[:24].copy()
        euro["e"] = 0
        want = want + (european(euro) - fd64(euro, x_dim, t_dim, scale, density))
    err = {}
    for solver in (kwg.SOLVER_AUTO, kwg.SOLVER_THOMAS):
        rc, p, st = price(o, kwg.params(t_dim=t_dim, x_dim=x_dim, scale=scale, density=density, solver=solver))
        assert rc == kwg.KWG_OK and (st == 0).all(), ctx.last_error()
        err[solver] = np.linalg.norm(p[:24] - want) / np.linalg.norm(want)
    tol = 3 * math.sqrt(t_dim - 1) * 2.0**-49 * (2 if bs else 1)
    assert err[kwg.SOLVER_AUTO] <= max(err[kwg.SOLVER_THOMAS], tol), err

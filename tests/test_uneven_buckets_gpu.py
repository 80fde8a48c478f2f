"""Uneven batches on the warp-per-PDE solvers: buckets that run on streams of their own."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 2), (33, 40), (64, 17), (65, 9), (128, 50), (250, 31), (512, 12), (777, 8), (1024, 20), (2048, 6), (2047, 5)]


def _batch(n, seed):
    import portfolio

    rng = np.random.default_rng(seed)
    o = portfolio.american_portfolio(n, seed=seed)
    shape = np.array(SHAPES, np.int32)[rng.integers(0, len(SHAPES), n)]
    return o, np.ascontiguousarray(shape[:, 0]), np.ascontiguousarray(shape[:, 1])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 37, 3000])
def test_buckets_match_uniform_calls(ctx, n, precision):
    """Every option against the call that has its grid alone (another padding of lanes and warps
    per PDE: FP64 to 1e-11, FP32 to 2e-7 of the strike), duplicates included, twice."""
    import kwg

    o, x, t = _batch(n, n)
    if n > 10:  # duplicates, across the caller's order and with other spots
        o[n // 2:n // 2 + 5], x[n // 2:n // 2 + 5], t[n // 2:n // 2 + 5] = o[:5], x[:5], t[:5]
        o["s"][n // 2] *= 1.01
    p = kwg.params(scale=5.0, density=math.inf, precision=precision)
    runs = [ctx.fd1d_price_uneven(o, x, t, p) for _ in range(2)]
    assert runs[0][0] == kwg.KWG_OK, ctx.last_error()
    assert np.array_equal(runs[0][1], runs[1][1], equal_nan=True) and np.array_equal(runs[0][2], runs[1][2])
    got, st = runs[0][1:]
    for xs, ts in set(zip(x.tolist(), t.tolist())):
        sel = (x == xs) & (t == ts)
        rc, want, st_w = ctx.fd1d_price(
            np.ascontiguousarray(o[sel]),
            kwg.params(scale=5.0, density=math.inf, precision=precision, x_dim=xs, t_dim=ts))
        assert rc == kwg.KWG_OK and np.array_equal(st[sel], st_w)
        ok = st_w == 0
        tol = 2e-7 if precision else 1e-11
        assert np.all(np.abs(got[sel][ok] - want[ok]) <= tol * o["k"][sel][ok])


def test_strict_names_the_callers_first_failure(ctx):
    """Failures in two buckets: strict mode reports the one that comes first in the caller's order, with
    and without a status array."""
    import kwg

    o, x, t = _batch(200, 5)
    x[:], t[:] = 128, 20
    x[120:], t[120:] = 2048, 6  # the heavier bucket runs first
    o["t"][150] = float("nan")
    o["z"][40] = -1.0
    p = kwg.params(scale=5.0, density=math.inf, strict=1)
    rc, prices, st = ctx.fd1d_price_uneven(o, x, t, p)
    assert rc != kwg.KWG_OK and "asset 40:" in ctx.last_error()
    assert np.flatnonzero(st).tolist() == [40, 150]
    again = np.empty(len(o))
    rc2 = kwg.lib().kwg_fd1d_price_uneven(ctx.ptr, o.ctypes.data, x.ctypes.data, t.ctypes.data, len(o),
                                          ctypes.byref(p), again.ctypes.data, None)
    assert rc2 == rc and np.array_equal(again, prices, equal_nan=True)

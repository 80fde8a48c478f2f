"""Device memory that an uneven call holds: rows for the distinct PDEs, not for the options."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_duplicates_take_no_rows(built, precision):
    """80000 options on 800 PDEs of 1000 and 2000 nodes: 10 MB of rows (1 GB without deduplication)."""
    import kwg
    import portfolio
    import torch

    n, per = 80000, 100
    key = np.arange(n) // per
    o = portfolio.american_portfolio(n // per, seed=1)[key]
    o["s"] = o["k"] * (0.9 + 0.2 * portfolio.uniforms(2, 9, n))
    x = np.where(key % 2 == 0, 2000, 1000).astype(np.int32)
    t = np.full(n, 4, np.int32)
    c = kwg.Context(0)
    try:
        prm = kwg.params(scale=5.0, density=math.inf, precision=precision)
        rc, want, _ = c.fd1d_price_uneven(o[::per].copy(), x[::per].copy(), t[::per].copy(), prm)  # module loading
        assert rc == kwg.KWG_OK
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        rc, p, st = c.fd1d_price_uneven(o, x, t, prm)
        assert rc == kwg.KWG_OK and (st == 0).all()
        assert free - torch.cuda.mem_get_info()[0] <= 128 << 20
        assert np.allclose(p[::per], want, rtol=1e-9 if precision == 0 else 1e-5, atol=0 if precision == 0 else 1e-5)
    finally:
        c.close()


def test_buckets_with_different_shares_of_duplicates(built):
    """The first bucket all duplicates, the others none (their buffers grow), then the other way round."""
    import kwg
    import portfolio

    n = 3000
    o = portfolio.american_portfolio(n, seed=5)
    x = np.repeat(np.array([1024, 60, 300], np.int32), n // 3)
    t = np.full(n, 12, np.int32)
    c, fresh = kwg.Context(0), kwg.Context(0)
    try:
        for precision in (0, 1):
            prm = kwg.params(scale=5.0, density=math.inf, precision=precision)
            for dup in ([0], [1, 2], [0, 1, 2], []):
                q = o.copy()
                for k in dup:
                    for f in ("t", "z", "r", "q", "w", "e"):
                        q[f][k * n // 3:(k + 1) * n // 3] = o[f][k * n // 3]
                rc, p, st = c.fd1d_price_uneven(q, x, t, prm)
                assert rc == kwg.KWG_OK, c.last_error()
                for k in range(3):
                    s = slice(k * n // 3, (k + 1) * n // 3)
                    rc, want, _ = fresh.fd1d_price(q[s].copy(), kwg.params(scale=5.0, density=math.inf, precision=precision,
                                                                         x_dim=int(x[s][0]), t_dim=12))
                    assert rc == kwg.KWG_OK
                    assert np.all(np.abs(p[s] - want) <= (2e-7 if precision else 1e-11) * q["k"][s])
    finally:
        c.close()
        fresh.close()

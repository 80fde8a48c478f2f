"""FP32 stepping over the time value: grids that fill the lanes and grids padded in front, the
payoff's kink between lanes, inside one and on two-node lanes, 1 to 4 warps per PDE."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP32 rounds the operator's coefficients by 2^-24, which moves a price by a few 1e-8 of the strike;
# 2e-7 leaves a factor of ten.
TOL = 2e-7


@pytest.mark.parametrize("density", [math.inf, 0.25])
@pytest.mark.parametrize("x_dim,warps", [
    (3, 0), (33, 0), (50, 0), (63, 1), (64, 1), (65, 1), (127, 1), (129, 1), (255, 4), (300, 2), (511, 1), (512, 4),
    (513, 2), (777, 1), (1023, 2), (1024, 1), (1024, 4), (1025, 2), (2047, 4), (2048, 2)])
def test_padding_and_kink(ctx, x_dim, warps, density):
    import kwg
    import kwor
    import portfolio

    n, t_dim = 12, 60
    o = portfolio.american_portfolio(n, seed=x_dim)
    o["e"][::4] = 0  # European: no floor anywhere
    p = kwg.params(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=density, precision=kwg.FP32, option_warps=warps)
    rc, got, st = ctx.fd1d_price(o, p)
    rc_ref, msg, want, st_ref = kwor.fd1d_price(o, t_dim=t_dim, x_dim=x_dim, scale=5.0, density=density)
    assert rc == kwg.KWG_OK and rc_ref == 0, msg
    assert (st == 0).all() and (st_ref == 0).all()
    assert np.max(np.abs(got - want) / o["k"]) <= TOL


@pytest.mark.parametrize("precision,tol", [(0, 1e-11), (1, TOL)])
@pytest.mark.parametrize("t_dim", [16, 40, 1500])
@pytest.mark.parametrize("x_dim", [51, 64, 128, 256, 512, 1024])
def test_reduction_levels(ctx, x_dim, t_dim, precision, tol):
    """Time steps from coarse to fine: all five levels of the separators' reduction down to one (FP64
    accuracy: 1e-11 of the strike, a tenth of the parity bar)."""
    import kwg
    import kwor
    import portfolio

    o = portfolio.american_portfolio(8, seed=t_dim)
    p = kwg.params(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=math.inf, precision=precision,
                   option_warps=1 if precision else 0)
    rc, got, st = ctx.fd1d_price(o, p)
    rc_ref, msg, want, st_ref = kwor.fd1d_price(o, t_dim=t_dim, x_dim=x_dim, scale=5.0, density=math.inf)
    assert rc == kwg.KWG_OK and rc_ref == 0, msg
    assert (st == 0).all() and (st_ref == 0).all()
    assert np.max(np.abs(got - want) / o["k"]) <= tol

"""Which FP64 solver KWG_SOLVER_AUTO takes at theta = 1/2: many PDEs of few nodes and few steps on ragged
uniform grids stream, all else runs on chip, in the uniform and the uneven call alike; batches with
many PDEs that pair arithmetic leaves over are stepped in FP64.  The routes are told apart by their bits (streaming
lanes and on-chip PDEs do not depend on their neighbours) and launches (pair arithmetic 3, FP64 on chip 2)."""
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


def drifting(n, share, seed=4):
    """`share` of the options with a drift of more than 0.3 half-widths of a grid at scale 5."""
    import portfolio

    o = portfolio.american_portfolio(n, seed=seed)
    k = portfolio.uniforms(seed, 40, n) < share
    o["z"][k], o["r"][k], o["q"][k], o["t"][k] = 0.03, 0.08, 0.0, 1.5
    o["t"][k] += np.arange(k.sum()) * 1e-4  # PDEs of their own
    o["s"] = o["k"]
    return o


@pytest.mark.parametrize("n,x_dim,t_dim,share,route", [
    (20000, 65, 40, 1.0, "stream"), (12000, 300, 12, 0.9, "stream"), (300, 512, 40, 0.1, "fp64"), (60, 1500, 20, 0.2, "fp64"),
    (2000, 256, 40, 1.0, "fp64"), (6000, 512, 60, 0.05, "pair")])
@pytest.mark.parametrize("entry", ["host", "bs"])
def test_batches_crossed_by_their_drift(built, entry, n, x_dim, t_dim, share, route):
    import kwg

    c = kwg.Context(0)
    try:
        o = drifting(n // 2 if entry == "bs" else n, share)
        call = c.fd1d_bs_price if entry == "bs" else c.fd1d_price
        kw = dict(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=math.inf)
        rc, p, st = call(o, kwg.params(**kw))
        assert rc == kwg.KWG_OK, c.last_error()
        launches = c.launch_count() - (entry == "bs")
        rc, want, wst = call(o, kwg.params(solver=kwg.SOLVER_THOMAS, **kw))
        assert rc == kwg.KWG_OK and np.array_equal(st, wst)
        ok = st == 0
        assert ok.all()
        assert np.max(np.abs(p - want) / np.maximum(1e-10 * np.abs(want), 1e-13 * o["k"])) <= 1.0
        if route == "stream":
            assert np.array_equal(p, want)
        else:
            assert not np.array_equal(p, want) and launches == (2 if route == "fp64" else 3)
    finally:
        c.close()


@pytest.mark.parametrize("n,share,streams", [(30000, 1.0, True), (30000, 0.02, False)])
def test_uneven_batches_crossed_by_their_drift(built, n, share, streams):
    import kwg

    c = kwg.Context(0)
    try:
        rng = np.random.default_rng(n)
        o = drifting(n, share)
        x, t = (rng.integers(*r, n).astype(np.int32) for r in ((90, 140), (20, 50)))
        got = {}
        for s in (kwg.SOLVER_AUTO, kwg.SOLVER_THOMAS, kwg.SOLVER_PCR):
            rc, got[s], _ = c.fd1d_price_uneven(o, x, t, kwg.params(scale=5.0, density=math.inf, solver=s))
            assert rc == kwg.KWG_OK, c.last_error()
        assert not np.array_equal(got[1], got[2])
        assert np.array_equal(got[0], got[1] if streams else got[2])
        assert np.max(np.abs(got[0] - got[1]) / np.maximum(1e-10 * np.abs(got[1]), 1e-13 * o["k"])) <= 1.0
    finally:
        c.close()


@pytest.mark.parametrize("n,x_dim,t_dim,share", [(20000, 65, 40, 1.0), (12000, 300, 12, 0.9), (300, 512, 40, 0.1),
                                                 (60, 1500, 20, 0.2), (6000, 512, 60, 0.05), (20000, 65, 40, 0.01)])
@pytest.mark.parametrize("dedup", [0, 1])
def test_device_calls_choose_as_host_calls(built, n, x_dim, t_dim, share, dedup):
    """Bit for bit, also when the next batch on the same buffers takes the other route."""
    import kwg
    import torch

    c = kwg.Context(0)
    try:
        prm = kwg.params(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=math.inf)
        prm.device_dedup = dedup
        price = torch.empty(n, dtype=torch.float64, device="cuda")
        status = torch.empty(n, dtype=torch.int32, device="cuda")
        for s in (share, 0.0, share):
            o = drifting(n, s)
            rc, want, wst = c.fd1d_price(o, kwg.params(t_dim=t_dim, x_dim=x_dim, scale=5.0, density=math.inf))
            assert rc == kwg.KWG_OK
            d = torch.from_numpy(o.view(np.uint8).copy()).cuda()
            torch.cuda.synchronize()
            rc = c.fd1d_price_device(d.data_ptr(), n, prm, price.data_ptr(), status.data_ptr(), 0)
            assert rc == kwg.KWG_OK, c.last_error()
            torch.cuda.synchronize()
            assert np.array_equal(price.cpu().numpy(), want) and np.array_equal(status.cpu().numpy(), wst)
    finally:
        c.close()


@pytest.mark.parametrize("n,x_dim,t_dim,density,fp64", [(40, 300, 100, 0.25, True), (40, 64, 40, math.inf, True),
                                                        (40, 128, 600, 0.25, True), (40, 300, 600, 0.25, False),
                                                        (40, 700, 40, 0.25, False), (40, 128, 40, math.inf, False)])
def test_small_control_variates_step_in_fp64(built, n, x_dim, t_dim, density, fp64):
    """Where the two solves' errors cancel better than pair arithmetic resolves (launches: FP64 on chip 2,
    pair arithmetic 3, and the control variate)."""
    import kwg
    import portfolio

    c = kwg.Context(0)
    try:
        o = portfolio.american_portfolio(n, seed=x_dim)
        got = {}
        for s in (kwg.SOLVER_AUTO, kwg.SOLVER_THOMAS):
            rc, got[s], st = c.fd1d_bs_price(o, kwg.params(t_dim=t_dim, x_dim=x_dim, scale=50.0 if density < 1 else 5.0,
                                                           density=density, solver=s))
            assert rc == kwg.KWG_OK and (st == 0).all()
            if s == kwg.SOLVER_AUTO:
                assert c.launch_count() == (3 if fp64 else 4)
        assert np.max(np.abs(got[0] - got[1]) / np.maximum(1e-10 * np.abs(got[1]), 1e-13 * o["k"])) <= 1.0
    finally:
        c.close()


def test_a_bucket_with_few_left_over_keeps_pair_arithmetic(built):
    """Buckets run side by side, so one PDE left over does not send a bucket of a thousand to FP64 stepping, as it would
    send a batch of its own (launches of an on-chip bucket: pair arithmetic 3, FP64 2)."""
    import kwg

    c = kwg.Context(0)
    try:
        o = drifting(1000, 0.0)
        o["z"][7], o["r"][7], o["q"][7], o["t"][7] = 0.03, 0.08, 0.0, 1.5
        x, t = np.full(1000, 200, np.int32), np.full(1000, 60, np.int32)
        prm = kwg.params(scale=5.0, density=math.inf)
        rc, p, st = c.fd1d_price_uneven(o, x, t, prm)
        assert rc == kwg.KWG_OK and (st == 0).all() and c.launch_count() == 3
        o["z"], o["r"], o["q"], o["t"] = 0.03, 0.08, 0.0, 1.5 + 1e-4 * np.arange(1000)
        rc, p, st = c.fd1d_price_uneven(o, x, t, kwg.params(scale=5.0, density=math.inf, solver=kwg.SOLVER_PCR))
        assert rc == kwg.KWG_OK and (st == 0).all() and c.launch_count() == 2
    finally:
        c.close()


@pytest.mark.parametrize("entry", ["host", "uneven", "device"])
def test_without_room_for_streaming_it_stays_on_chip(built, entry):
    """2.1 million PDEs of 2048 nodes: 310 GB for the streaming solver, which the cost model names, 34 GB on chip."""
    import kwg
    import torch

    n, x_dim = 2100000, 2048
    o = drifting(3000, 1.0)[np.arange(n) % 3000]
    o["t"] += 1e-9 * np.arange(n)  # PDEs of their own
    torch.cuda.empty_cache()
    total = torch.cuda.mem_get_info()[1]
    if not 40 * 10**9 < total < 305 * 10**9:
        pytest.skip("sized for a device of 298 GB")
    c = kwg.Context(0)
    try:
        kw = dict(scale=5.0, density=math.inf)
        if entry == "uneven":
            rc, p, st = c.fd1d_price_uneven(o, np.full(n, x_dim), np.full(n, 3), kwg.params(**kw))
        elif entry == "host":
            rc, p, st = c.fd1d_price(o, kwg.params(t_dim=3, x_dim=x_dim, **kw))
        else:
            d = torch.from_numpy(o.view(np.uint8).copy()).cuda()
            price, status = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
            rc = c.fd1d_price_device(d.data_ptr(), n, kwg.params(t_dim=3, x_dim=x_dim, **kw), price.data_ptr(),
                                     status.data_ptr(), 0)
            torch.cuda.synchronize()
            p, st = price.cpu().numpy(), status.cpu().numpy()
        assert rc == kwg.KWG_OK, c.last_error()
        assert (st == 0).all()
        pick = np.arange(0, n, 6007)
        rc, want, _ = c.fd1d_price(o[pick], kwg.params(t_dim=3, x_dim=x_dim, solver=kwg.SOLVER_THOMAS, **kw))
        assert rc == kwg.KWG_OK and np.max(np.abs(p[pick] - want) / np.maximum(1e-10 * np.abs(want), 1e-13 * o["k"][pick])) <= 1.0
    finally:
        c.close()

"""The surrogate's pricing kernel at the edges of its tile pipeline, and its analytic base price."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(built):
    import kwg

    s = kwg.Surrogate(0)
    yield s
    s.close()


def _device(o):
    import torch

    return torch.from_numpy(o.view(np.uint8).copy()).cuda()


@pytest.mark.parametrize("tiles,rows", [(0, 127), (1, 0), (152, 1), (2 * 152, 0), (3 * 152, 127), (5 * 152 + 1, 1)])
def test_tiles_and_slots(net, tiles, rows):
    """Each block walks 128-option tiles through two slots: a lone tile, one to six tiles per
    block (both slots reused), ragged ends; against the layer-by-layer path (same FP32 network,
    same base price: 1e-12 of the strike)."""
    import mlp_oracle as mo
    import portfolio
    import torch

    n = 128 * tiles + rows
    net.set_params(mo.random_params(5), mo.BOX_LO, mo.BOX_HI, 250.0)
    o = portfolio.american_portfolio(n, seed=n)
    o["e"][1::7] = 0
    d_o = _device(o)
    price = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    f = torch.empty((n, 5), dtype=torch.float32, device="cuda")
    inside, inside2 = (torch.full((n,), 7, dtype=torch.uint8, device="cuda") for _ in range(2))
    base = torch.empty(n, dtype=torch.float64, device="cuda")
    y = torch.empty(n, dtype=torch.float32, device="cuda")
    net.price_device(d_o.data_ptr(), n, price.data_ptr(), inside.data_ptr())
    net.featurize(d_o.data_ptr(), n, f.data_ptr(), inside2.data_ptr(), base.data_ptr())
    net.forward(f.data_ptr(), n, y.data_ptr())
    torch.cuda.synchronize()
    want = base.cpu().numpy() + o["k"] * (y.cpu().numpy() / np.float32(250.0)).astype(np.float64)
    intrinsic = np.maximum(0.0, o["w"] * (o["s"] - o["k"]))
    want = np.where(o["e"] != 0, np.maximum(want, intrinsic), want)
    assert np.max(np.abs(price.cpu().numpy() - want) / o["k"]) <= 1e-12
    assert torch.equal(inside, inside2)


@pytest.mark.parametrize("case", ["wide", "small rates", "zero rates", "negative rates", "small vol"])
def test_base_price_matches_oracle(net, case):
    """Barone-Adesi-Whaley base price against the FP64 bisection, within 2e-6 of the strike: FP32 carries
    the root and the premium (16 roundings of 2^-23)."""
    import mlp_oracle as mo
    import portfolio
    import torch

    n, rng = 20000, np.random.default_rng(3)
    o = portfolio.american_portfolio(n, seed=11)
    if case == "wide":
        o["z"], o["t"] = np.exp(rng.uniform(-4, 0.5, n)), np.exp(rng.uniform(-6, 2.5, n))
        o["r"], o["q"] = rng.uniform(0, 0.15, n), rng.uniform(0, 0.15, n)
        o["k"] = o["s"] * np.exp(rng.uniform(-2, 2, n))
    elif case == "small rates":
        o["r"], o["q"] = np.exp(rng.uniform(-25, -2, n)), np.exp(rng.uniform(-25, -2, n))
    elif case == "zero rates":
        o["r"], o["q"] = (np.where(rng.random(n) < 0.3, 0.0, o[f]) for f in ("r", "q"))
    elif case == "negative rates":
        o["r"], o["q"] = rng.uniform(-0.05, 0.1, n), rng.uniform(-0.05, 0.1, n)
    else:
        o["z"], o["t"] = np.exp(rng.uniform(-12, -4, n)), 1.0
    d_o = _device(o)
    base = torch.empty(n, dtype=torch.float64, device="cuda")
    net.featurize(d_o.data_ptr(), n, 0, 0, base.data_ptr())
    torch.cuda.synchronize()
    assert np.max(np.abs(base.cpu().numpy() - mo.baw(o)) / o["k"]) <= 2e-6

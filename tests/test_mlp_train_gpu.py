"""The one-kernel minibatch gradients at the edges of its 64-row tiles: one row, a full and an
over-full tile, and more tiles than SMs (a second tile on one CTA), against the NumPy oracle that
applies the same BF16 roundings, per weight and bias block within 5e-3 of its norm and the
loss within 1e-4, as the 300-row test of test_mlp_gpu.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 152 * 64 + 1])
def test_gradient_tiles(built, n):
    import torch

    import kwg
    import mlp_oracle as mo

    net = kwg.Surrogate(0, seed=3)
    try:
        p = mo.random_params(n)
        net.set_params(p)
        rng = np.random.default_rng(n)
        f = rng.uniform(-1.0, 1.0, (n, 5)).astype(np.float32)
        t = rng.normal(size=n).astype(np.float32)
        fl = np.where(np.arange(n) % 4 == 3, rng.normal(size=n), -mo.NO_FLOOR).astype(np.float32)
        x = np.zeros((n, mo.W))
        x[:, :5] = f
        lo, go = mo.gradients(p, x, t.astype(np.float64), floor=fl.astype(np.float64))
        d_f, d_t, d_fl = (torch.from_numpy(a).cuda() for a in (f, t, fl))
        d_g = torch.empty(kwg.MLP_PARAMS, dtype=torch.float32, device="cuda")
        for _ in range(2):  # the second call starts from the first one's sums
            loss = net.gradients(d_f.data_ptr(), d_t.data_ptr(), n, d_g.data_ptr(), d_fl.data_ptr())
            g = d_g.cpu().numpy().astype(np.float64)
            assert abs(loss - lo) <= 1e-4 * lo
            W, NW = mo.W, mo.N_WEIGHTS
            for l in range(mo.LAYERS):
                for a, b in ((l * W * W, (l + 1) * W * W), (NW + l * W, NW + (l + 1) * W)):
                    assert np.linalg.norm(g[a:b] - go[a:b]) <= 5e-3 * np.linalg.norm(go[a:b]), (l, a)
    finally:
        net.close()

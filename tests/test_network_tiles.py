"""The network's fused kernels at the edges of their tiles: one tile per
minibatch (fewer chunks than the weight gradients' ring is deep), several
tiles, minibatches past the first, and inference at row counts around a tile.
Against the CPU restatement with the same bf16 roundings, at the tolerances
of tests/test_mlp.py (gradients 1e-2 of each block's norm, losses 1e-3,
values 1e-2 of the targets' scale: activations rounded to bf16, 2^-9, through
three layers)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from test_mlp import _blocks, _peak_data  # noqa: E402


@pytest.mark.parametrize("batch,minibatches", [(128, 3), (256, 1), (640, 2)])
def test_gradients_per_minibatch(cub, ctx, batch, minibatches):
    import numpy as np
    import mlp_oracle as M

    E, S = 3, batch * minibatches
    x, y = _peak_data(E, S, batch)
    net = cub.Mlp(E, S, batch=batch, seed=7)
    net.set_data(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"))
    p = net.params()
    for b in range(minibatches):
        loss, g = net.grad(b)
        part = slice(b * batch, (b + 1) * batch)
        for e in range(E):
            ys = (y[e] / np.abs(y[e]).max())[part]
            l_ref, g_ref = M.grad(p[e], x[e, part], ys)
            assert abs(loss[e] - l_ref) <= 1e-3 * l_ref
            for name, (i, j) in _blocks().items():
                ref = g_ref[i:j]
                d = np.linalg.norm(g[e, i:j] - ref) / max(np.linalg.norm(ref), 1e-30)
                assert d <= 1e-2, (b, e, name, d)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 5000])
def test_inference_row_counts(cub, ctx, n):
    import numpy as np
    import mlp_oracle as M

    E, S = 2, 256
    x, y = _peak_data(E, S, 3)
    net = cub.Mlp(E, S, batch=128, seed=3)
    net.set_data(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"))
    net.train(3, 1e-3)
    p = net.params()
    xt = np.random.default_rng(n).uniform(0, 1, (E, n, 7))
    g = net.eval(torch.tensor(xt, device="cuda")).cpu().numpy()
    for e in range(E):
        scale = np.abs(y[e]).max()
        ref, _ = M.forward(p[e], xt[e])
        assert np.abs(g[e] - scale * ref).max() <= 1e-2 * scale

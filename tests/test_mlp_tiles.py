"""The network's kernels at the edges of their tiles: the forward pass over 128-sample tiles,
also from inputs that are not 16-byte aligned, and the training pass over 32-sample tiles,
also with more tiles than blocks."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _net(seed):
    from myfvcomcode_b200.engine import Mlp
    rng = np.random.default_rng(seed)
    p = (0.2 * rng.standard_normal(mo.NPAR)).astype(np.float32)
    net = Mlp(seed=0)
    net.set_params(p)
    return net, p, rng


@pytest.mark.parametrize("n,offset", [(1, 0), (127, 0), (128, 1), (129, 0), (1000, 3), (57000, 0)])
def test_forward_tiles(n, offset):
    import torch
    net, p, rng = _net(n)
    x = (2.0 * rng.standard_normal((n, mo.MI))).astype(np.float32)
    buf = torch.zeros(n * mo.MI + offset, dtype=torch.float32, device="cuda")
    buf[offset:] = torch.from_numpy(x.reshape(-1)).cuda()
    out = torch.zeros((n + 1, mo.MO), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    net.forward(buf.data_ptr() + 4 * offset, n, out.data_ptr())
    ref, _ = mo.forward(p.astype(np.float64), x.astype(np.float64))
    got = out.cpu().numpy()
    assert np.abs(got[:n] - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    assert np.all(got[n] == 0.0)
    net.close()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 9473, 20001])
def test_gradient_tiles(n):
    import torch
    net, p, rng = _net(n)
    x = rng.standard_normal((n, mo.MI)).astype(np.float32)
    y = rng.standard_normal((n, mo.MO)).astype(np.float32)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    torch.cuda.synchronize()
    loss, g = net.loss_grad(dx.data_ptr(), dy.data_ptr(), n)
    loss_o, g_o = mo.loss_grad(p.astype(np.float64), x, y)
    assert abs(loss - loss_o) <= 1e-5 * loss_o
    assert np.abs(g - g_o).max() <= 2e-5 * np.abs(g_o).max()
    net.close()

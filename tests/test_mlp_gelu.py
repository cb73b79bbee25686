"""The derivative of the closure network's GELU in FP32 against 64 bits, unit by unit, from
well below zero to where the function is the identity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gelu_d(z):
    c = np.sqrt(2.0 / np.pi)
    t = np.tanh(c * (z + 0.044715 * z ** 3))
    return 0.5 * (1.0 + t) + 0.5 * z * (1.0 - t * t) * c * (1.0 + 3.0 * 0.044715 * z * z)


def _gelu(z):
    return 0.5 * z * (1.0 + np.tanh(np.sqrt(2.0 / np.pi) * (z + 0.044715 * z ** 3)))


@pytest.mark.parametrize("lo,hi", [(-0.5, 0.5), (0.5, 2.0), (2.0, 4.0), (4.0, 6.0), (6.0, 12.0)])
def test_gradient_through_one_unit(lo, hi):
    # One sample, unit j of the first layer at z_j (its bias), unit j of the second at
    # gelu(z_j)/64, every one with weight 1 in the first output; the target is far off, so that
    # the output's error is exact to a rounding.  The gradient of bias j is that error times
    # gelu'(gelu(z_j)/64)/64 times gelu'(z_j).  Two derivatives of two to three units in the last
    # place and four roundings: below 16 x 2^-24 = 1e-6 of it.
    import torch
    from myfvcomcode_b200.engine import Mlp
    net = Mlp(seed=1)
    z = np.linspace(lo, hi, 64).astype(np.float32)
    w2 = np.zeros((64, 64), np.float32)
    np.fill_diagonal(w2, 1.0 / 64.0)
    w3 = np.zeros((3, 64), np.float32)
    w3[0] = 1.0
    p = np.concatenate([np.zeros(512, np.float32), z, w2.ravel(), np.zeros(64, np.float32), w3.ravel(),
                        np.zeros(3, np.float32)])
    net.set_params(p)
    x = torch.zeros((1, 8), device="cuda")
    y = torch.tensor([[-4096.0, 0.0, 0.0]], device="cuda")
    torch.cuda.synchronize()
    _, g = net.loss_grad(x.data_ptr(), y.data_ptr(), 1)
    z = z.astype(np.float64)
    h = _gelu(z) / 64.0
    want = 2.0 / 3.0 * (_gelu(h).sum() + 4096.0) * _gelu_d(h) / 64.0 * _gelu_d(z)
    got = g[512:576].astype(np.float64)
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
    net.close()

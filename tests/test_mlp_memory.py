"""A batch that finds no room for its blocks' gradients fails; the network works on afterwards."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_batch_without_room():
    import torch
    from myfvcomcode_b200.engine import FvgError, Mlp
    a, b = Mlp(seed=1), Mlp(seed=1)
    n = 32 * 296
    x = torch.randn((n, 8), device="cuda")
    y = torch.randn((n, 3), device="cuda")
    torch.cuda.synchronize()
    first = a.loss_grad(x.data_ptr(), y.data_ptr(), 32)
    cuda = ctypes.CDLL("libcuda.so.1")
    held = []
    for size in (1 << 30, 1 << 20, 1 << 16):  # every byte that a later allocation could have
        while True:
            p = ctypes.c_uint64()
            if cuda.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)):
                break
            held.append(p)
    try:
        with pytest.raises(FvgError):
            a.loss_grad(x.data_ptr(), y.data_ptr(), n)
    finally:
        for p in held:
            cuda.cuMemFree_v2(p)
    again = a.loss_grad(x.data_ptr(), y.data_ptr(), 32)
    assert again[0] == first[0] and np.array_equal(again[1], first[1])
    g, w = a.loss_grad(x.data_ptr(), y.data_ptr(), n), b.loss_grad(x.data_ptr(), y.data_ptr(), n)
    assert g[0] == w[0] and np.array_equal(g[1], w[1])
    a.close()
    b.close()

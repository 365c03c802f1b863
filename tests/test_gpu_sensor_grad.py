"""The sensor's loss gradient at the edges of its tiles of 64 samples and over
several tiles a block, against the CPU restatement of the network in 64 bits.
A gradient is a sum of up to n terms in FP32: the bound is eps times the square
root of the number of sequential additions a sum can see (tile length, tiles of
a block, blocks: at most 64 + 6 + 296), with a factor four, of the norm."""
import ctypes

import numpy as np
import pytest

from artracfd_b200 import abi, sensor
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu
TOL = 4 * np.finfo(np.float32).eps * np.sqrt(64 + 6 + 296)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 64 * 296, 64 * 296 * 5 + 17])
def test_gradient_at_tile_edges(n):
    import torch
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 10)).astype(np.float32)
    y = (rng.random(n) < 0.3).astype(np.float32)
    p = sensor.init_params(3)
    loss_ref, grad_ref = mlp_oracle.loss_and_grad(p, X, y, 2.5)
    lib = abi.load_library()
    vp = ctypes.c_void_p
    dp, dx, dy = (torch.tensor(a, device="cuda") for a in (p, X, y))
    g = torch.zeros(p.size, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    abi.check(lib.acfd_mlp_grad(vp(dp.data_ptr()), vp(dx.data_ptr()), vp(dy.data_ptr()), n, 2.5, vp(g.data_ptr()),
                                vp(loss.data_ptr()), None), lib)
    torch.cuda.synchronize()
    got = g.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - grad_ref) <= TOL * np.linalg.norm(grad_ref)
    assert abs(float(loss.item()) - loss_ref) <= TOL * abs(loss_ref)

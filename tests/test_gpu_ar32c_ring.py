"""The FP32 filter's slice ring (one slot more than the order's slices, the next
slice's halo brought in early) at its shortest and longest, on surfaces of several
tiles and of fewer slices than the order, against the FP64 filter."""
import numpy as np
import pytest

import arma_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [
    ((1, 40, 70), (4, 4, 4)), ((2, 40, 70), (1, 3, 3)), ((9, 33, 65), (1, 1, 1)),
    ((9, 33, 65), (1, 16, 13)), ((9, 33, 65), (2, 1, 4)), ((30, 20, 40), (16, 2, 3)),
    ((20, 50, 100), (13, 16, 2)), ((7, 100, 37), (3, 4, 13)), ((120, 17, 33), (2, 2, 2)),
])
def test_ring(shape, order):
    import torch
    rng = np.random.default_rng(sum(shape) + sum(order))
    phi = rng.uniform(-1.0, 1.0, order)
    phi.flat[0] = 0.0
    phi *= 0.9 / max(np.abs(phi).sum(), 1.0)  # a contraction: rounding stays local
    eps = rng.standard_normal(shape).astype(np.float32)
    z32 = torch.from_numpy(eps.copy()).cuda()
    z64 = torch.from_numpy(eps.astype(np.float64)).cuda()
    with A.Context(0) as ctx:
        ctx.ar_filter(phi, shape, A.FP32C, z32.data_ptr())
        ctx.ar_filter(phi, shape, A.FP64, z64.data_ptr())
        ctx.synchronize()
    d = (z32.double() - z64).cpu().numpy()
    # storage in FP32 (6e-8) amplified by at most 1 / (1 - 0.9)
    assert np.sqrt(np.mean(d * d)) <= 1e-6 * np.sqrt(np.mean(z64.cpu().numpy() ** 2))

"""The FP64 filter's tiles of two cells per thread, which a batch with enough work
takes: every tap count they hold and the widths beyond, windows of one row and of
many, ragged surfaces, bit for bit the result of each surface by itself."""
import os

import numpy as np
import pytest

import arma_b200 as A
from arma_b200 import capi

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("shape", [(19, 48, 48), (23, 45, 50), (30, 33, 31), (1, 64, 70)])
def test_batch_equals_single(shape):
    import torch
    mt = A.mt_file_read(os.path.join(ROOT, "arma_b200", "data", "mt.dat"), 0)
    rng = np.random.default_rng(sum(shape))
    fits = []
    for k in range(120):
        order = ((1, 3, 4)[k % 3], (1, 2, 5, 10)[k % 4], k % 12 + 1)
        phi = rng.uniform(-1.0, 1.0, order)
        phi.flat[0] = 0.0
        fits.append(phi * (0.9 / max(np.abs(phi).sum(), 1.0)))  # a contraction
    out = torch.zeros((2, len(fits)) + shape, dtype=torch.float64, device="cuda")
    surf = [[capi.make_surface(shape, p, 1.0, 0.0, mt, 50 + k, out[b, k].data_ptr())
             for k, p in enumerate(fits)] for b in range(2)]
    with A.Context(0) as ctx:
        ctx.batch_generate(surf[0], A.FP64)
        for one in surf[1]:
            ctx.batch_generate([one], A.FP64)
        ctx.synchronize()
    got = out.cpu().numpy()
    assert np.isfinite(got).all() and np.abs(got).max() > 0.0
    assert np.array_equal(got[0], got[1])

"""The FP32 filter's CTAs per SM by the batch's concurrency: surfaces of 128 tiles,
so that one, some and many can run at once, give the same bits as one CTA per SM."""
import os

import numpy as np
import pytest

import arma_b200 as A
from arma_b200 import capi

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [1, 2, 4, 9])
def test_same_bits(n):
    import torch
    mt = A.mt_file_read(os.path.join(ROOT, "arma_b200", "data", "mt.dat"), 0)
    shape = (40, 256, 256)
    phi, var = A.ar_fit_analytic(A.ACF_STANDING, (3, 3, 3), 1.5, 0.8, [0.05] * 3, [0.5, 0.5])
    got = []
    with A.Context(0) as ctx:
        for per_sm in (0, 1):
            t = ctx.tuning()
            t.ar_ctas_per_sm = per_sm
            ctx.set_tuning(t)
            out = torch.empty((n,) + shape, dtype=torch.float32, device="cuda")
            ctx.batch_generate([capi.make_surface(shape, phi, var, 1.5, mt, 7 + k,
                                                  out[k].data_ptr()) for k in range(n)], A.FP32C)
            ctx.synchronize()
            got.append(out.cpu().numpy())
    assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])

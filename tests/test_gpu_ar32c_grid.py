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


@pytest.mark.parametrize("shape", [(20, 95, 1925), (20, 970, 190), (4, 700, 1110), (3, 16, 6000),
                                   (3, 3000, 32)])
def test_more_tiles_than_run_at_once(shape):
    """Wide, tall and square grids of tiles against the FP64 filter."""
    import torch
    rng = np.random.default_rng(sum(shape))
    phi = rng.uniform(-1.0, 1.0, (3, 4, 5))
    phi.flat[0] = 0.0
    phi *= 0.9 / np.abs(phi).sum()  # a contraction: rounding stays local
    eps = rng.standard_normal(shape).astype(np.float32)
    z32 = torch.from_numpy(eps.copy()).cuda()
    z64 = torch.from_numpy(eps.astype(np.float64)).cuda()
    with A.Context(0) as ctx:
        t = ctx.tuning()
        t.ar_ctas_per_sm = 1
        ctx.set_tuning(t)
        ctx.ar_filter(phi, shape, A.FP32C, z32.data_ptr())
        ctx.ar_filter(phi, shape, A.FP64, z64.data_ptr())
        ctx.synchronize()
    d = (z32.double() - z64).cpu().numpy()
    # storage in FP32 (6e-8) amplified by at most 1 / (1 - 0.9)
    assert np.sqrt(np.mean(d * d)) <= 1e-6 * np.sqrt(np.mean(z64.cpu().numpy() ** 2))


@pytest.mark.parametrize("shape", [(30, 288, 576), (30, 90, 1900), (30, 1300, 100)])
def test_keeping_pace_has_the_same_bits(shape):
    """Tiles of many taps, two or three to an SM and all at once, which hold back for
    the tiles below them, against one CTA per SM."""
    import torch
    rng = np.random.default_rng(sum(shape))
    phi = rng.uniform(-1.0, 1.0, (8, 7, 8))
    phi.flat[0] = 0.0
    phi *= 0.9 / np.abs(phi).sum()
    eps = torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda()
    got = []
    with A.Context(0) as ctx:
        for per_sm in (1, 2, 3, 0):
            t = ctx.tuning()
            t.ar_ctas_per_sm = per_sm
            ctx.set_tuning(t)
            z = eps.clone()
            torch.cuda.synchronize()
            ctx.ar_filter(phi, shape, A.FP32C, z.data_ptr())
            ctx.synchronize()
            got.append(z)
    assert torch.isfinite(got[0]).all() and all(torch.equal(got[0], g) for g in got[1:])

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


@pytest.mark.parametrize("order,per_sm", [((16, 13, 9), 2), ((16, 13, 12), 2), ((11, 10, 10), 3),
                                          ((13, 16, 5), 3), ((11, 11, 8), 3)])
def test_ring_without_the_slot_ahead(order, per_sm):
    """Orders whose ring gives up its extra slot for another CTA on the SM, alone and
    beside small orders that keep theirs: the bits of one CTA per SM, which has it."""
    import torch
    from arma_b200 import capi
    rng = np.random.default_rng(sum(order))
    shapes = [(20, 40, 100), (33, 50, 37), (5, 70, 70)]
    orders = [order, (2, 3, 4), order]
    phis = []
    for o in orders:
        phi = rng.uniform(-1.0, 1.0, o)
        phi.flat[0] = 0.0
        phis.append(phi * 0.9 / np.abs(phi).sum())
    mt = A.mt19937_params()
    got = []
    with A.Context(0) as ctx:
        for n in (1, per_sm):
            t = ctx.tuning()
            t.ar_ctas_per_sm = n
            ctx.set_tuning(t)
            out = [torch.zeros(s, dtype=torch.float32, device="cuda") for s in shapes]
            torch.cuda.synchronize()
            ctx.batch_generate([capi.make_surface(s, p, 1.0, 0.0, mt, 3 + k, z.data_ptr())
                                for k, (s, p, z) in enumerate(zip(shapes, phis, out))], A.FP32C)
            ctx.synchronize()
            got.append(out)
    assert all(torch.isfinite(a).all() and torch.equal(a, b) for a, b in zip(*got))

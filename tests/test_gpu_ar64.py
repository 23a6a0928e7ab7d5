"""The FP64 AR filter's tile wavefront against the oracle's sequential loop:
bit for bit at the edges of its tiles, for every width of order, for the tile
shapes it chooses among and for batches of surfaces."""
import numpy as np
import pytest

import arma_b200 as A
import oracle as O
from arma_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with A.Context(0) as c:
        yield c


def model(order, rng, lag0=0.0):
    """Coefficients of absolute sum 0.9: the filter's values stay bounded."""
    phi = rng.uniform(-1.0, 1.0, order)
    phi.flat[0] = 0.0
    phi *= 0.9 / max(np.abs(phi).sum(), 1.0)
    phi.flat[0] = lag0
    return phi


def run(ctx, eps, phi):
    import torch
    z = torch.from_numpy(eps.copy()).cuda()
    ctx.ar_filter(phi, eps.shape, A.FP64, z.data_ptr())
    ctx.synchronize()
    return z.cpu().numpy()


# tile edges in x and u = x + y (tiles of 8 or 16 rows by 8 or 16 columns), thin
# surfaces, halos wider than a tile, orders of every tap count and the largest
@pytest.mark.parametrize("shape,order", [
    ((5, 8, 16), (3, 3, 3)), ((4, 9, 17), (2, 3, 3)), ((7, 16, 15), (4, 2, 5)),
    ((3, 17, 1), (2, 4, 3)), ((6, 1, 33), (3, 3, 7)), ((40, 1, 1), (9, 2, 2)),
    ((6, 33, 31), (1, 1, 1)), ((6, 20, 20), (1, 1, 5)), ((6, 20, 20), (1, 5, 1)),
    ((20, 12, 13), (5, 1, 1)), ((9, 30, 25), (2, 10, 9)), ((9, 40, 37), (3, 16, 2)),
    ((9, 26, 60), (3, 2, 16)), ((5, 35, 40), (11, 11, 11)), ((4, 24, 33), (12, 12, 12)),
    ((3, 40, 39), (16, 16, 16)), ((20, 18, 18), (16, 3, 13)), ((8, 18, 22), (3, 4, 14)),
    ((8, 18, 22), (3, 4, 15)), ((8, 18, 22), (3, 4, 6)), ((8, 18, 22), (3, 4, 8)),
    ((33, 70, 90), (4, 5, 10)), ((12, 260, 200), (3, 4, 4)),
])
def test_tiles_bit_exact(ctx, shape, order):
    rng = np.random.default_rng(sum(shape) + 7 * sum(order))
    phi = model(order, rng)
    eps = rng.standard_normal(shape)
    assert np.array_equal(run(ctx, eps, phi), O.ar_filter(eps, phi))


# more tiles than the device holds at once: handed out by anti-diagonals
@pytest.mark.parametrize("shape,order", [
    ((2, 800, 810), (2, 3, 3)), ((1, 60, 9000), (1, 2, 4)), ((1, 9000, 60), (1, 4, 2)),
    ((3, 700, 500), (1, 16, 1)), ((2, 300, 290), (2, 12, 12)), ((12, 330, 340), (3, 10, 10)),
])
def test_more_tiles_than_run_at_once(ctx, shape, order):
    rng = np.random.default_rng(sum(shape))
    phi, eps = model(order, rng), rng.standard_normal(shape)
    assert np.array_equal(run(ctx, eps, phi), O.ar_filter(eps, phi))


def test_planes_of_more_than_2_31_points(ctx):
    """Noise in the last corner of a plane whose points have 64-bit offsets: the
    filter there is that of the corner alone."""
    import torch
    n, corner = 46400, 100
    rng = np.random.default_rng(9)
    phi, eps = model((1, 4, 3), rng), rng.standard_normal((1, corner, corner))
    z = torch.zeros((1, n, n), dtype=torch.float64, device="cuda")
    z[0, n - corner:, n - corner:] = torch.from_numpy(eps[0]).cuda()
    torch.cuda.synchronize()
    ctx.ar_filter(phi, z.shape, A.FP64, z.data_ptr())
    assert not z[0, :n - corner].any() and not z[0, :, :n - corner].any()
    got = z[0, n - corner:, n - corner:].cpu().numpy()
    del z
    torch.cuda.empty_cache()
    assert np.array_equal(got, O.ar_filter(eps, phi)[0])


def test_own_lag_and_overwritten_noise(ctx):
    """A coefficient at lag (0, 0, 0) multiplies the point's own noise."""
    rng = np.random.default_rng(5)
    phi, eps = model((3, 4, 3), rng, lag0=0.25), rng.standard_normal((9, 19, 21))
    assert np.array_equal(run(ctx, eps, phi), O.ar_filter(eps, phi))


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_coefficients_that_are_not_finite(ctx, bad):
    """The reference's sum is truncated at the array's start: an infinite
    coefficient reaches only the points that have its lag."""
    rng = np.random.default_rng(6)
    phi, eps = model((2, 3, 3), rng), rng.standard_normal((5, 9, 10))
    phi[1, 2, 1] = bad
    with np.errstate(all="ignore"):
        ref = O.ar_filter(eps, phi)
    got = run(ctx, eps, phi)
    assert np.isfinite(got).any() and np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize("shape,order", [((1, 1, 1), (16, 16, 16)), ((2, 30, 40), (9, 4, 4)),
                                         ((20, 3, 40), (3, 8, 4)), ((20, 40, 2), (3, 4, 11)),
                                         ((1, 50, 50), (5, 6, 7))])
def test_order_longer_than_the_surface(ctx, shape, order):
    """Lags that no point has, infinite ones among them, are not part of any sum."""
    rng = np.random.default_rng(8)
    phi, eps = model(order, rng), rng.standard_normal(shape)
    outside = np.logical_or.reduce([i >= n for i, n in zip(np.indices(order), shape)])
    phi[outside] = np.inf
    ref = O.ar_filter(eps, phi)
    assert np.isfinite(ref).all() and np.array_equal(run(ctx, eps, phi), ref)


def test_noise_that_is_not_finite(ctx):
    rng = np.random.default_rng(7)
    phi, eps = model((3, 3, 4), rng), rng.standard_normal((6, 20, 37))
    eps[2, 9, 20] = np.inf
    with np.errstate(all="ignore"):
        ref = O.ar_filter(eps, phi)
    assert np.array_equal(run(ctx, eps, phi), ref, equal_nan=True)


@pytest.mark.parametrize("count", [3, 40])
def test_batch_bit_exact(ctx, count):
    """Surfaces of mixed shape and order in one call (few: the narrow tiles;
    many: the wide ones) against the same surfaces one by one, and the first
    against the oracle's filter of the same noise."""
    import torch
    rng = np.random.default_rng(count)
    mt = A.mt19937_params()
    shapes = [tuple(int(v) for v in (rng.integers(5, 30), rng.integers(6, 70),
                                     rng.integers(6, 70))) for _ in range(count)]
    phis = [model(tuple(int(v) for v in rng.integers(1, 9, 3)), rng) for _ in range(count)]

    def surfaces(bufs):
        return [capi.make_surface(s, p, 0.7, 0.0, mt, 90 + k, b.data_ptr())
                for k, (s, p, b) in enumerate(zip(shapes, phis, bufs))]

    bufs = [torch.zeros(s, dtype=torch.float64, device="cuda") for s in shapes]
    ctx.batch_generate(surfaces(bufs), A.FP64)
    alone = [torch.zeros_like(b) for b in bufs]
    for s in surfaces(alone):
        ctx.batch_generate([s], A.FP64)
    assert all(torch.equal(a, b) for a, b in zip(bufs, alone))
    n = int(np.prod(shapes[0]))
    eps = torch.zeros(n, dtype=torch.float64, device="cuda")
    ctx.white_noise(mt, 90, float(np.sqrt(0.7)), n, A.FP64, eps.data_ptr())
    ctx.synchronize()
    ref = O.ar_filter(eps.cpu().numpy().reshape(shapes[0]), phis[0])
    assert np.array_equal(bufs[0].cpu().numpy(), ref)

"""The velocity window's own exponential and its ranges, the division by
constants in the passes and the split of spectra and depths, against the
oracle: finite and infinite depth, z at the bottom, depths where the window
underflows, many depths, and slices of every kernel (one CTA, a CTA pair,
banded passes) with prime and odd sides."""
import numpy as np
import pytest

import arma_b200 as A
import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with A.Context(0) as c:
        yield c


@pytest.mark.parametrize("shape,depth,zs", [
    ((3, 32, 16), 12.0, [0.0, -0.5, -1.0, -3.0, -12.0]),
    ((3, 128, 128), np.inf, [0.0, -1.0, -2.0, -4.0, -8.0]),
    ((3, 256, 256), 40.0, [0.0, -40.0]),
    ((3, 64, 64), np.inf, [0.0, -100.0, -115.0, -300.0]),   # exponents around -350 and far below
    ((3, 64, 64), 600.0, [0.0, -200.0, -599.0]),
    ((2, 37, 53), 7.0, [0.0, -7.0]),
    ((2, 976, 5), np.inf, [0.0, -2.0]),
    ((2, 4, 1024), np.inf, [-1.0]),
    ((3, 200, 100), np.inf, [0.0, -1.0, -90.0]),
])
@pytest.mark.parametrize("high_amplitude", [False, True])
def test_window_and_split(ctx, shape, depth, zs, high_amplitude):
    rng = np.random.default_rng(sum(shape))
    # smooth slices, so that the steep form's slopes stay below one; not smooth in
    # time, where the mean of three slices would leave no derivative
    zeta = rng.standard_normal(shape)
    for axis in (1, 2):
        zeta = (zeta + np.roll(zeta, 1, axis) + np.roll(zeta, 2, axis)) / 3.0
    delta = (0.5, 0.8, 1.25)
    tidx = list(range(shape[0]))
    solve = O.velocity_high_amplitude if high_amplitude else O.velocity_linear
    ref = solve(zeta, delta, depth, zs, tidx)
    assert np.isfinite(ref).all()
    scale = np.abs(ref).max()
    # the bars of the other solver tests: FFT rounding in FP64 and FP32
    for prec, dt, tol in [(A.FP64, torch.float64, 1e-9), (A.FP32C, torch.float32, 2e-4)]:
        z = torch.tensor(zeta, dtype=dt, device="cuda")
        out = torch.zeros(ref.shape, dtype=dt, device="cuda")
        ctx.velocity_linear(z.data_ptr(), shape, prec, delta, depth, zs, tidx, out.data_ptr(),
                            high_amplitude=high_amplitude)
        got = out.cpu().numpy().astype(np.float64)
        assert np.abs(got - ref).max() <= tol * scale, (prec, np.abs(got - ref).max() / scale)


def test_more_depths_than_a_grid_dimension(ctx):
    """65540 depths of one small slice: the last ones as a call of their own has them."""
    rng = np.random.default_rng(3)
    z = torch.tensor(rng.standard_normal((3, 32, 16)), dtype=torch.float32, device="cuda")
    zs = np.linspace(0.0, -4.0, 65540)

    def run(levels):
        out = torch.full((1, len(levels), 32, 16), np.nan, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.velocity_linear(z.data_ptr(), (3, 32, 16), A.FP32C, (1.0, 1.0, 1.0), np.inf,
                            list(levels), [1], out.data_ptr())
        ctx.synchronize()
        return out

    whole = run(zs)
    assert torch.isfinite(whole).all()
    for part in (slice(0, 3), slice(65533, 65540)):
        assert torch.equal(whole[:, part], run(zs[part]))


@pytest.mark.parametrize("shape", [(3, 32, 16), (2, 37, 53), (3, 256, 256)])
def test_depth_that_is_not_a_number(ctx, shape):
    """Every entry of the window is then non-finite and becomes 0, as in the reference."""
    rng = np.random.default_rng(4)
    zeta = rng.standard_normal(shape)
    ref = O.velocity_linear(zeta, (1.0, 1.0, 1.0), np.nan, [-1.0, -2.0], [1])
    assert not ref.any()
    for prec, dt in [(A.FP64, torch.float64), (A.FP32C, torch.float32)]:
        z = torch.tensor(zeta, dtype=dt, device="cuda")
        out = torch.ones(ref.shape, dtype=dt, device="cuda")
        torch.cuda.synchronize()
        ctx.velocity_linear(z.data_ptr(), shape, prec, (1.0, 1.0, 1.0), np.nan, [-1.0, -2.0], [1],
                            out.data_ptr())
        ctx.synchronize()
        assert not out.cpu().numpy().any()

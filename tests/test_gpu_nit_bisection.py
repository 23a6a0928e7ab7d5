"""The table and the cubics of the per-point bisection against the same call on so
few points that it has neither (every F(c) evaluated): the same bits, for smooth,
sharp and non-monotone distributions, every stopping rule, odd intervals and values
that are not finite."""
import numpy as np
import pytest

import arma_b200 as A

pytestmark = pytest.mark.gpu

SKEW, GRAM = A.NIT_SKEW_NORMAL, A.NIT_GRAM_CHARLIER


@pytest.fixture(scope="module")
def ctx():
    with A.Context(0) as c:
        yield c


@pytest.mark.parametrize("dist,params,interval,eps,max_iter", [
    (SKEW, [0.0, 1.0, 1.499], (-10.0, 10.0), 1e-6, 100),
    (SKEW, [0.0, 1.0, 1.499], (-10.0, 10.0), 1e-10, 100),
    (SKEW, [0.0, 1.0, 1.499], (-10.0, 10.0), 1e-300, 70),   # to the last bit
    (SKEW, [0.3, 0.5, -4.0], (-6.0, 5.0), 1e-8, 100),
    (SKEW, [0.0, 1.0, 60.0], (-10.0, 10.0), 1e-9, 100),     # a narrow feature
    (SKEW, [0.0, 1.0, 0.0], (0.0, 1.0), 1e-6, 100),         # most roots outside
    (GRAM, [0.1, 3.2], (-10.0, 10.0), 1e-6, 100),
    (GRAM, [-0.2, 3.0], (-5.0, 5.0), 1e-4, 100),
    (GRAM, [1.5, 6.0], (-10.0, 10.0), 1e-9, 100),           # not monotone
    (SKEW, [0.0, 1.0, 1.499], (5.0, -5.0), 1e-6, 20),       # reversed
    (SKEW, [0.0, 1.0, 1.499], (-1e300, 1e300), 1e-6, 100),
    (GRAM, [0.1, 3.2], (-10.0, 10.0), 1e-6, 7),             # stops inside the table
])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_same_as_evaluating_every_point(ctx, dist, params, interval, eps, max_iter, dtype):
    import torch
    rng = np.random.default_rng(3)
    v = rng.normal(0.0, 1.2, 70000).astype(dtype)
    v[:6] = [np.nan, np.inf, -np.inf, 0.0, 9.0, -9.0]
    prec = A.FP64 if dtype == "float64" else A.FP32C
    big = torch.from_numpy(v.copy()).cuda()

    def apply(z):
        ctx.nit_apply(dist, params, 1.2, A.NIT_BISECTION, z.numel(), prec, z.data_ptr(),
                      interval=interval, eps=eps, max_iter=max_iter)
        ctx.synchronize()

    torch.cuda.synchronize()
    apply(big)
    for at in [0, 8, 16, 1000, 33333, 69992] + list(range(40000, 44000, 40)):
        few = torch.from_numpy(v[at:at + 8].copy()).cuda()
        torch.cuda.synchronize()
        apply(few)
        assert np.array_equal(few.cpu().numpy(), big[at:at + 8].cpu().numpy(), equal_nan=True), at


@pytest.mark.parametrize("params,interval", [
    ([1e6, -3e5], (-10.0, 10.0)), ([1e9, 0.0], (0.9, 1.1)), ([-1e9, 3.0], (-1.02, -0.97)),
    ([3e6, 0.0], (0.99, 1.01)), ([1e12, 0.0], (0.5, 1.2)), ([3e6, 0.0], (0.9999, 1.0001)),
    ([0.0, 4e5], (1.7, 1.75)),
])
def test_values_far_above_one(ctx, params, interval):
    """A Gram-Charlier CDF of such skewness and kurtosis rounds at its own size, not
    at that of a probability: to the last bit of the bracket."""
    import torch
    rng = np.random.default_rng(5)
    v = rng.normal(0.0, 1.2, 1 << 18)
    big = torch.from_numpy(v.copy()).cuda()
    few = torch.from_numpy(v.copy()).cuda()
    torch.cuda.synchronize()

    def apply(z):
        ctx.nit_apply(GRAM, params, 1.2, A.NIT_BISECTION, z.numel(), A.FP64, z.data_ptr(),
                      interval=interval, eps=1e-300, max_iter=200)

    apply(big)
    for part in few.split(256):  # too few points for cubics: every F(c) evaluated
        apply(part)
    ctx.synchronize()
    assert torch.equal(big, few)

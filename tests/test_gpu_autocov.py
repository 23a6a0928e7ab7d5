"""The device auto-covariance's mixed-radix bands against numpy's FFT in FP64:
every radix, primes on every axis, sides of 1 and the largest, odd numbers of
lines, bands with a ragged last column."""
import numpy as np
import pytest

import arma_b200 as A

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with A.Context(0) as c:
        yield c


@pytest.mark.parametrize("shape", [
    (1, 1, 1), (1, 1, 7), (1, 5, 1), (9, 1, 1), (2, 2, 2), (3, 4, 5), (8, 7, 6), (1, 3, 1024),
    (1024, 2, 3), (2, 1024, 5), (3, 1021, 2), (1021, 1, 3), (1, 3, 1021), (4, 6, 67), (49, 27, 25),
    (13, 11, 121), (64, 128, 31), (22, 38, 94), (30, 1, 127), (16, 16, 1000),
])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_against_numpy(ctx, shape, dtype):
    import torch
    w = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dtype)
    f = np.fft.fftn(w.astype(np.float64))
    ref = np.fft.ifftn(np.abs(f) ** 2).real / w.size
    src = torch.from_numpy(w).cuda()
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    ctx.auto_covariance(src.data_ptr(), shape, A.FP64 if dtype == "float64" else A.FP32C,
                        out.data_ptr())
    ctx.synchronize()
    # out(0, 0, 0) is the mean square, the largest value; direct sums of 1021
    # terms round to about 1e-13 of it
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))

"""The FP32 filter's tap rows: every tap count, rows of coefficients with and
without low parts (all, some, none), slices whose rows are and are not 16-byte
aligned, against the FP64 filter."""
import numpy as np
import pytest

import arma_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("py", range(1, 14))
@pytest.mark.parametrize("low", ["all", "some", "none"])
def test_rows(py, low):
    import torch
    order = (3, 4, py)
    rng = np.random.default_rng(py)
    phi = rng.uniform(-1.0, 1.0, order)
    phi.flat[0] = 0.0
    phi *= 0.9 / max(np.abs(phi).sum(), 1.0)  # a contraction: rounding stays local
    exact = phi.astype(np.float32).astype(np.float64)
    if low == "none":
        phi = exact
    elif low == "some":
        phi[:, 1::2] = exact[:, 1::2]
    with A.Context(0) as ctx:
        for shape in [(9, 18, 64), (9, 33, 70)]:
            n = int(np.prod(shape))
            eps = rng.standard_normal(n).astype(np.float32)
            z64 = torch.from_numpy(eps.astype(np.float64)).cuda()
            ctx.ar_filter(phi, shape, A.FP64, z64.data_ptr())
            got = []
            for offset in (0, 1):  # in floats: rows on and off 16-byte boundaries
                z32 = torch.zeros(n + offset, dtype=torch.float32, device="cuda")
                z32[offset:] = torch.from_numpy(eps).cuda()
                torch.cuda.synchronize()
                ctx.ar_filter(phi, shape, A.FP32C, z32.data_ptr() + 4 * offset)
                ctx.synchronize()
                got.append(z32[offset:].clone())
            assert torch.equal(got[0], got[1])
            d = (got[0].double() - z64).cpu().numpy()
            # storage in FP32 (6e-8) amplified by at most 1 / (1 - 0.9)
            assert np.sqrt(np.mean(d * d)) <= 1e-6 * np.sqrt(np.mean(z64.cpu().numpy() ** 2))

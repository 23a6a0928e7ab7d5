"""The bounded waits of the AR filters: the self-test starves a tile of the FP32
and of the FP64 filter's own kernels, and a filter's error word is read before
the call returns."""
import numpy as np
import pytest

import arma_b200 as A
from arma_b200 import capi

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_selftest_runs_the_filters_kernels():
    with A.Context(0) as ctx:
        ctx.set_profiling(True)
        with pytest.raises(capi.ArmaError) as e:
            ctx.selftest_wait()
        assert e.value.code == -4
        assert ctx.profile("ar32c")[1] == 1 and ctx.profile("ar64")[1] == 1
        # no error is left for the next call
        z = torch.ones((4, 20, 40), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.ar_filter(np.full((1, 1, 2), 0.25), z.shape, A.FP64, z.data_ptr())
        ctx.synchronize()
        assert torch.isfinite(z).all()


@pytest.mark.parametrize("precision,dtype", [(A.FP64, torch.float64), (A.FP32C, torch.float32)])
def test_filter_has_been_checked_when_it_returns(precision, dtype):
    """The caller's own stream has nothing left to do."""
    with A.Context(0) as ctx:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        z = torch.zeros((600, 64, 64), dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):
            ctx.ar_filter(np.zeros((6, 6, 6)), z.shape, precision, z.data_ptr())
            assert stream.query()

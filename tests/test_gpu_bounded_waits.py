"""The bounded waits of the AR filters: a filter's error word is read before the
call returns."""
import numpy as np
import pytest

import arma_b200 as A

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


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

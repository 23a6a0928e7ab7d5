"""Two contexts on two host threads: calls whose kernels take very different amounts
of shared memory, side by side.  What a kernel may take is an attribute of the
function on the device, which both contexts share."""
import threading

import numpy as np
import pytest

import arma_b200 as A

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CALLS = 600


def both(make_small, make_large, calls=CALLS):
    """make_*(ctx) -> a call; each repeated on a thread of its own."""
    failures = []
    start = threading.Barrier(2)

    def work(make):
        try:
            with A.Context(0) as ctx:
                call = make(ctx)
                call()
                ctx.synchronize()
                start.wait(60)
                for k in range(calls):
                    call()
                    if k % 16 == 15:
                        ctx.synchronize()
                ctx.synchronize()
        except Exception as e:  # noqa: BLE001 (any failure of a thread is the test's)
            failures.append(e)
            start.abort()

    torch.cuda.init()
    threads = [threading.Thread(target=work, args=(m,)) for m in (make_small, make_large)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def autocov(shape):
    def make(ctx):
        w = torch.ones(shape, dtype=torch.float64, device="cuda")
        out = torch.zeros_like(w)
        torch.cuda.synchronize()
        return lambda: ctx.auto_covariance(w.data_ptr(), shape, A.FP64, out.data_ptr())
    return make


def test_auto_covariance():
    both(autocov((4, 4, 4)), autocov((3, 1021, 4)))

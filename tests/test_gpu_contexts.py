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


def fp32_filter(order):
    def make(ctx):
        z = torch.zeros((2, 8, 8), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return lambda: ctx.ar_filter(np.zeros(order), z.shape, A.FP32C, z.data_ptr())
    return make


def test_fp32_filter():
    both(fp32_filter((1, 1, 1)), fp32_filter((16, 13, 13)))


def words(params):
    def make(ctx):
        out = torch.zeros(1 << 19, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return lambda: ctx.mt_genrand(params, 1, 1 << 19, out.data_ptr())
    return make


def test_jumps():
    short, long = A.mt19937_params(), A.mt19937_params()
    short.nn, short.mm = 16, 8
    both(words(short), words(long))


def potentials(shape, precision, dtype):
    def make(ctx):
        z = torch.zeros(shape, dtype=dtype, device="cuda")
        out = torch.zeros((1, 2) + shape[1:], dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        return lambda: ctx.velocity_linear(z.data_ptr(), shape, precision, (1.0, 1.0, 1.0), np.inf,
                                           [0.0, -1.0], [1], out.data_ptr())
    return make


@pytest.mark.parametrize("precision,dtype,large", [
    (A.FP64, torch.float64, (3, 1000, 100)), (A.FP32C, torch.float32, (3, 120, 130)),
    (A.FP32C, torch.float32, (3, 1000, 1000)),
])
def test_velocity(precision, dtype, large):
    both(potentials((3, 5, 6), precision, dtype), potentials(large, precision, dtype))

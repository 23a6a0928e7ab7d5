"""The FP64 moving-average filter by matrix instructions: time lags on both sides of
its rule, numbers of taps with every remainder by four, several launches of one
order, ragged surfaces, against the oracle's direct sum."""
import numpy as np
import pytest

import arma_b200 as A
import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [
    ((9, 17, 65), (4, 3, 3)), ((9, 17, 65), (5, 3, 3)), ((8, 16, 64), (5, 1, 8)),
    ((7, 15, 63), (5, 1, 7)), ((17, 33, 70), (6, 1, 9)), ((30, 20, 9), (20, 2, 5)),
    ((5, 3, 130), (9, 5, 5)), ((1, 40, 40), (5, 4, 4)), ((12, 18, 30), (6, 30, 21)),
    ((20, 9, 100), (32, 10, 10)),
])
def test_against_direct_sum(shape, order):
    rng = np.random.default_rng(sum(shape) + sum(order))
    theta = rng.uniform(-1.0, 1.0, order)
    eps = rng.standard_normal(shape)
    e = torch.tensor(eps, device="cuda")
    z = torch.full(shape, np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with A.Context(0) as ctx:
        ctx.ma_filter(theta, shape, A.FP64, e.data_ptr(), z.data_ptr())
        ctx.synchronize()
    # each side sums P products in some order: P 2^-53 of the sum of magnitudes
    bound = 2 * theta.size * 2.0 ** -53 * (1.0 + np.abs(theta).sum()) * np.abs(eps).max()
    assert np.max(np.abs(z.cpu().numpy() - O.ma_filter(eps, theta))) <= bound


# tap counts that four does not divide and taps of single columns, on both sides
@pytest.mark.parametrize("shape,order", [
    ((20, 17, 65), (15, 3, 3)), ((20, 17, 65), (16, 3, 3)), ((9, 17, 65), (5, 5, 2)),
    ((9, 33, 30), (8, 10, 1)), ((9, 33, 30), (32, 8, 1)),
])
def test_sides_of_the_rule(shape, order):
    test_against_direct_sum(shape, order)


def test_noise_that_is_not_finite_stays_where_it_reaches():
    """An infinity in slice 5 meets, in the scalar form, the time steps 4 and later
    of its block: the steps before it keep their values."""
    shape, order = (24, 20, 70), (6, 3, 4)
    rng = np.random.default_rng(8)
    theta = rng.uniform(-1.0, 1.0, order)
    eps = rng.standard_normal(shape)
    got = []
    with A.Context(0) as ctx:
        for bad in (False, True):
            e = torch.tensor(eps, device="cuda")
            if bad:
                e[5, 7, 30] = np.inf
            z = torch.full(shape, np.nan, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ctx.ma_filter(theta, shape, A.FP64, e.data_ptr(), z.data_ptr())
            ctx.synchronize()
            got.append(z.cpu().numpy())
    bound = 2 * theta.size * 2.0 ** -53 * (1.0 + np.abs(theta).sum()) * np.abs(eps).max()
    assert np.max(np.abs(got[0][:4] - got[1][:4])) <= bound
    assert np.isposinf(got[1][5, 7, 30])
    reached = np.zeros(shape, bool)
    reached[:, 7:7 + order[1], 30:30 + order[2]] = True
    assert np.max(np.abs(got[0] - got[1])[~reached]) <= bound

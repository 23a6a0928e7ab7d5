"""The dcmt word stream where it is cut into segments, by one CTA or one warp per
segment, and for state sizes at the edges of the jump kernel's passes: equal to
the oracle's sequential generator bit for bit."""
import os

import numpy as np
import pytest

import arma_b200 as A
import oracle as O

pytestmark = pytest.mark.gpu

DATA = os.path.join(os.path.dirname(os.path.abspath(A.__file__)), "data", "mt.dat")
WHOLE, SEG = 1 << 18, 1 << 16  # longest uncut stream, shortest segment


@pytest.fixture(scope="module")
def ctx():
    with A.Context(0) as c:
        yield c


def shaped(nn, mm, rr, aaa):
    """A parameter set of any shape (its period need not be full)."""
    p = A.mt19937_params()
    p.nn, p.mm, p.rr, p.aaa, p.i = nn, mm, rr, aaa, nn
    p.umask = (0xffffffff << rr) & 0xffffffff
    p.lmask = 0xffffffff ^ p.umask
    return p


def check(ctx, p, seed, n, offset=0):
    import torch
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    ctx.mt_genrand(p, seed, n, out.data_ptr(), offset=offset)
    ctx.synchronize()
    ref = O.mt_genrand(O.MtParams.from_buffer_copy(p), seed, offset + n)[offset:]
    assert np.array_equal(out.cpu().numpy().view(np.uint32), ref)


@pytest.mark.parametrize("n,offset", [
    (1, 0), (1247, 0), (1248, 0), (1249, 0), (5000, 1247), (WHOLE, 0), (WHOLE + 1, 0),
    (5 * SEG + 3, 7), (100, 6 * SEG - 50), (SEG, 4 * SEG), (37 * SEG + 311, 2 * SEG + 5),
])
def test_cuts_of_a_committed_set(ctx, n, offset):
    check(ctx, A.mt_file_read(DATA, 5), 99, n, offset)


# one and several passes over the window (672 words each), shapes with nn = 2 mm
# down to a few slots, chunks longer than a block, MT19937
@pytest.mark.parametrize("nn,mm,rr", [(16, 8, 3), (6, 3, 0), (640, 320, 31), (672, 300, 1),
                                      (673, 336, 9), (1391, 695, 15), (624, 397, 31)])
@pytest.mark.parametrize("n", [3000, 7 * SEG + 11])
def test_shapes(ctx, nn, mm, rr, n):
    check(ctx, shaped(nn, mm, rr, 0x9908b0df), 4, n)


# windows too short for the four-step recurrence, over several jumps
@pytest.mark.parametrize("nn,mm,rr", [(2, 1, 3), (4, 2, 1), (6, 3, 1)])
def test_shortest_windows(ctx, nn, mm, rr):
    check(ctx, shaped(nn, mm, rr, 0x9908b0df), 4, 7 * SEG + 11)


@pytest.mark.parametrize("n", [1 << 19, 5 << 18])
def test_state_too_large_to_jump(ctx, n):
    """A state whose jump does not fit in shared memory: one sequential segment."""
    check(ctx, shaped(2000, 1000, 5, 0x9908b0df), 4, n)


def test_many_segments_by_warp(ctx):
    """More than six segments per SM: 900 streams of 2^18 words and one longer,
    through a batch's noise of two surfaces (the longer one cut)."""
    import torch
    from arma_b200 import capi
    mt = A.mt_file_read(DATA, 2)
    shapes = [(8, 90, 100)] * 900 + [(30, 160, 100)]
    phi = np.zeros((1, 1, 1))
    bufs = [torch.zeros(s, dtype=torch.float64, device="cuda") for s in shapes]
    ctx.batch_generate([capi.make_surface(s, phi, 1.0, 0.0, mt, 5 + k, b.data_ptr())
                        for k, (s, b) in enumerate(zip(shapes, bufs))], A.FP64)
    for k in (0, 899, 900):
        ref = O.white_noise(O.MtParams.from_buffer_copy(mt), 5 + k, 1.0, int(np.prod(shapes[k])))
        got = bufs[k].cpu().numpy().ravel()
        # log() may differ from the CPU's by one ulp
        assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-300)) <= 4e-16

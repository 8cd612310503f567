"""float32 stride-1 convolution in runs of planes and, for 16 gathered channels, on the tensor cores in three bfloat16 pieces: band
depths around the runs and windows, base planes that fit a window or not, all forms; values that the pieces cannot hold."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu


def _case(seed, B, H, W, D, Cin, Cout, spread):
    rng = np.random.default_rng(seed)
    r = lambda *s: rng.standard_normal(s).astype(np.float32)
    bp = rng.integers(0, spread + 1, (B, H, W, 1)).astype(np.int32)
    return r(B, H, W, D, Cin), r(3, 3, 3, Cin, Cout), bp, r(B, H, W, D, Cout)


cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("D,spread", [(1, 2), (3, 0), (4, 9), (5, 60), (7, 7), (7, 8), (10, 4), (11, 19), (11, 300), (24, 6), (25, 3), (64, 2)])
@pytest.mark.parametrize("chans", [(16, 16), (16, 32), (32, 16), (8, 16), (32, 8), (8, 8)])
def test_against_the_oracle(D, spread, chans):
    Cin, Cout = chans
    images, filters, bp, og = _case(D + spread, 2, 9, 21, D, Cin, Cout, spread)
    defv = 0.5
    want = oracle.sparse_conv3d_fwd(images, filters, defv, bp)
    ig_w, fg_w, _ = oracle.sparse_conv3d_bwd(images, filters, defv, bp, og)
    out = ops.sparse_conv3d_forward(cuda(images), cuda(filters), defv, cuda(bp))
    ig, fg, dg = ops.sparse_conv3d_backward(cuda(images), cuda(filters), defv, cuda(bp), cuda(og))
    # 27 * channels products of order one, summed in 24 bits: some units of 2^-24 times the root of the number of terms
    assert helpers.rel_err(out.cpu().numpy(), want) <= 3e-6
    assert helpers.rel_err(ig.cpu().numpy(), ig_w) <= 3e-6
    # 2*9*21*D products: the root of their number times 2^-24, against the largest sum of as many
    assert helpers.rel_err(fg.cpu().numpy(), fg_w) <= 3e-6 and float(dg) == 0.0
    coarse = og                                            # the transposed op at strides 1: gather form with the real default
    t_w = oracle.sparse_conv3d_transpose_fwd(coarse, filters, defv, bp, images.shape[1:4])
    t = ops.sparse_conv3d_transpose_forward(cuda(coarse), cuda(filters), defv, cuda(bp), images.shape[1:4])
    assert helpers.rel_err(t.cpu().numpy(), t_w) <= 3e-6
    assert _lib.lib().chop_umma_timeouts() == 0


@pytest.mark.parametrize("spread", [3, 60])   # one window, and staged column by column
@pytest.mark.parametrize("what", ["images", "filters"])
def test_values_that_the_pieces_cannot_hold(what, spread):
    images, filters, bp, _ = _case(9, 1, 7, 19, 9, 16, 16, spread)
    run = lambda i, f: ops.sparse_conv3d_forward(cuda(i), cuda(f), 0.0, cuda(bp)).cpu().numpy()
    plain = run(images, filters)
    tiny = np.float32(2.0 ** -70)                          # exact scaling: the same result, scaled
    scaled = run(images * tiny, filters) if what == "images" else run(images, filters * tiny)
    assert helpers.rel_err(scaled.astype(np.float64) / float(tiny), plain) <= 3e-6
    x = (images if what == "images" else filters).copy()
    x[0, 2, 2, 1, 3] = np.inf
    x[0, 0, 1, 2, 4] = np.nan
    got = run(x, filters) if what == "images" else run(images, x)
    _lib.set_tuning("tile", 2)
    try:
        want = run(x, filters) if what == "images" else run(images, x)
    finally:
        _lib.set_tuning("tile", 1)
    if what == "images":
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        assert np.array_equal(got[np.isinf(got)], want[np.isinf(got)])
        ok = np.isfinite(want)
        assert helpers.rel_err(got[ok], want[ok]) <= 3e-6
    else:   # where a tap of a zero default value meets them depends on the kernel: test_sparse_pieces_gpu.py
        assert not np.isfinite(got[..., 3]).all() and np.isnan(got[..., 4]).any()
        ok = np.isfinite(got) & np.isfinite(want)
        assert helpers.rel_err(got[ok], want[ok]) <= 3e-6

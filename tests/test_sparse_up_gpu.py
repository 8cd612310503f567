"""The transposed convolution and the strided image gradient with every coarse voxel staged once (strides 2 along rows and columns, 1 or
2 along depth, 8 or 16 produced channels; bfloat16, and float32 in three bfloat16 pieces): band depths at the ends of the windows, base planes that need one and several passes,
negative ones, odd images, tiles that the image does not divide, a zero and a non-zero default value, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


@pytest.mark.parametrize("dtype", [bf, torch.float32])
@pytest.mark.parametrize("strides", [(2, 2, 2), (2, 2, 1)])
@pytest.mark.parametrize("shape", [(2, 11, 37, 9), (1, 5, 18, 1), (1, 8, 35, 10), (1, 7, 12, 11), (1, 6, 20, 24)])
@pytest.mark.parametrize("spread", [0, 6, 200])
@pytest.mark.parametrize("chans,default", [((16, 16), 0.0), ((16, 16), 0.75), ((8, 8), 0.75), ((16, 32), 0.75), ((8, 16), 0.0)])
def test_against_the_oracle(strides, shape, spread, chans, default, dtype):
    Cin, Cout = chans
    B, H, W, D = shape
    rng = np.random.default_rng(D + spread)
    rnd = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(dtype)
    coarse = [-(-n // s) for n, s in zip((H, W, D), strides)]
    images, filters, fine = rnd(B, *coarse, Cout), rnd(3, 3, 3, Cin, Cout) * 0.25, rnd(B, H, W, D, Cin)
    bp = rng.integers(-3, spread - 2, (B, H, W, 1)).astype(np.int32)
    f = lambda t: t.float().numpy()
    up = ops.sparse_conv3d_transpose_forward(images.cuda(), filters.cuda(), default, torch.from_numpy(bp).cuda(), (H, W, D), strides)
    ig = ops.sparse_conv3d_backward(fine.cuda(), filters.cuda(), default, torch.from_numpy(bp).cuda(), images.cuda(), strides)[0]
    want = oracle.sparse_conv3d_transpose_fwd(f(images), f(filters), default, bp, (H, W, D), strides)
    ig_w = oracle.sparse_conv3d_bwd(f(fine), f(filters), default, bp, f(images), strides)[0]
    # bfloat16: results rounded to half a unit in the last place of eight bits, relative to the largest; float32: some units of 2^-24
    # times the root of the number of terms
    bound = 2.0 ** -8 if dtype == bf else 3e-6
    assert helpers.rel_err(up.float().cpu().numpy(), want) <= bound
    assert helpers.rel_err(ig.float().cpu().numpy(), ig_w) <= bound
    assert _lib.lib().chop_umma_timeouts() == 0


@pytest.mark.parametrize("strides", [(2, 2, 2), (2, 2, 1)])
def test_values_that_the_pieces_cannot_hold(strides):
    H, W, D = 9, 38, 9
    rng = np.random.default_rng(4)
    coarse = [-(-n // s) for n, s in zip((H, W, D), strides)]
    images = rng.standard_normal((1, *coarse, 16)).astype(np.float32)
    filters = rng.standard_normal((3, 3, 3, 16, 16)).astype(np.float32)
    bp = torch.from_numpy(rng.integers(0, 7, (1, H, W, 1)).astype(np.int32)).cuda()
    run = lambda i, f: ops.sparse_conv3d_transpose_forward(torch.from_numpy(i).cuda(), torch.from_numpy(f).cuda(), 0.0, bp, (H, W, D),
                                                           strides).cpu().numpy()
    plain, tiny = run(images, filters), np.float32(2.0 ** -70)   # exact scaling: the same result, scaled
    for i, f in ((images * tiny, filters), (images, filters * tiny)):
        assert helpers.rel_err(run(i, f).astype(np.float64) / float(tiny), plain) <= 3e-6
    images[0, 2, 5, 1, 3], images[0, 1, 12, 2, 4] = np.inf, np.nan
    got = run(images, filters)
    _lib.set_tuning("tile", 2)
    try:
        want = run(images, filters)
    finally:
        _lib.set_tuning("tile", 1)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert helpers.rel_err(got[ok], want[ok]) <= 3e-6

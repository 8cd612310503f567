"""The stride-1 tensor-core convolution that stages every voxel once per tile: band depths at the ends of its two windows, base
planes that fit one window, just miss it (a second pass) and fit none (staged column by column), images that the tiles do not
divide, all channel pairs, forward and image gradient, a non-zero default value."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


def _base(kind, rng, B, H, W, slack):
    """slack: planes that base_plane may vary by within a tile of one pass."""
    r, c = np.indices((H, W))
    if kind == "flat":
        bp = np.full((H, W), 3)
    elif kind == "fits":
        bp = rng.integers(0, slack + 1, (H, W))
    elif kind == "two passes":
        bp = rng.integers(0, slack + 2, (H, W))
    elif kind == "slope":
        bp = 2 * c + r
    else:
        bp = rng.integers(-40, 2000, (H, W))
    return np.broadcast_to(bp[None, :, :, None], (B, H, W, 1)).astype(np.int32)


@pytest.mark.parametrize("D,kind", [(1, "fits"), (9, "flat"), (9, "fits"), (9, "two passes"), (9, "slope"), (9, "rough"), (10, "two passes"),
                                    (11, "fits"), (11, "rough"), (17, "slope"), (24, "two passes"), (24, "rough"), (25, "fits")])
@pytest.mark.parametrize("chans", [(16, 16), (8, 32), (32, 8)])
def test_against_the_oracle(D, kind, chans):
    Cin, Cout = chans
    B, H, W = (1, 101, 163) if D <= 10 else (2, 13, 19)   # 16-row windows are used from 16000 pixels on
    rng = np.random.default_rng(D + len(kind))
    rnd = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(bf)
    images, filters, og = rnd(B, H, W, D, Cin), rnd(3, 3, 3, Cin, Cout) * 0.25, rnd(B, H, W, D, Cout)
    defv = 0.75
    bp = _base(kind, rng, B, H, W, (16 if D <= 10 else 32) - 2 - D)
    dev = lambda t: t.to("cuda")
    out = ops.sparse_conv3d_forward(dev(images), dev(filters), defv, dev(torch.from_numpy(bp)))
    ig = ops.sparse_conv3d_backward(dev(images), dev(filters), defv, dev(torch.from_numpy(bp)), dev(og))[0]
    f = lambda t: t.float().numpy()
    want = oracle.sparse_conv3d_fwd(f(images), f(filters), defv, bp)
    ig_w = oracle.sparse_conv3d_bwd(f(images), f(filters), defv, bp, f(og))[0]
    # results rounded to bfloat16: half a unit in the last place of eight bits, relative to the largest
    assert helpers.rel_err(out.float().cpu().numpy(), want) <= 2.0 ** -8
    assert helpers.rel_err(ig.float().cpu().numpy(), ig_w) <= 2.0 ** -8
    assert _lib.lib().chop_umma_timeouts() == 0

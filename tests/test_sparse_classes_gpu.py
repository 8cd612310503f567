"""The strided tensor-core kernels that work by (row, column) residue class and with swapped roles: strides with one, two
and more classes, classes without taps (stride 4), odd image sizes, bands that do not divide by the depth stride, a zero
and a non-zero default value, 16 / 32 channels on either side."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers
from tests.test_oracle_sparse import make_case, make_transpose_case

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


def _t(a, dt=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    return t.to(dt) if dt is not None else t


def _round(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(bf).float().numpy()


STRIDES = [(2, 2, 2), (1, 2, 2), (3, 2, 1), (2, 1, 3), (4, 4, 2), (1, 1, 2)]


@pytest.mark.parametrize("strides", STRIDES)
@pytest.mark.parametrize("chans,default", [((16, 16), 0.0), ((16, 16), None), ((32, 16), None), ((16, 32), 0.0), ((32, 32), None)])
def test_transposed_convolution(strides, chans, default):
    Cin, Cout = chans
    B, H, W, D = 2, 11, 13, 7
    images, filters, defv, bp = make_transpose_case(51, B, H, W, D, Cin, Cout, (3, 3, 3), strides, dtype=np.float32,
                                                    default=default)
    images, filters, defv = _round(images), _round(filters * 0.3), float(_round(np.array([defv]))[0])
    want = oracle.sparse_conv3d_transpose_fwd(images, filters, defv, bp, (H, W, D), strides, (1, 1, 1), np.float32)
    og = _round(np.random.default_rng(52).uniform(-1, 1, want.shape))
    ig_w, fg_w = oracle.sparse_conv3d_transpose_bwd(images, filters, defv, bp, (H, W, D), og, strides, (1, 1, 1), False,
                                                    np.float32)
    out = ops.sparse_conv3d_transpose_forward(_t(images, bf), _t(filters, bf), defv, _t(bp), (H, W, D), strides)
    ig, fg = ops.sparse_conv3d_transpose_backward(_t(images, bf), _t(filters, bf), defv, _t(bp), (H, W, D), _t(og, bf), strides)
    assert helpers.rel_err(out.float().cpu().numpy(), want) <= 1e-2
    assert helpers.rel_err(ig.float().cpu().numpy(), ig_w) <= 1e-2
    assert helpers.rel_err(fg.cpu().numpy(), fg_w) <= 1e-5
    assert _lib.lib().chop_umma_timeouts() == 0


@pytest.mark.parametrize("strides", STRIDES)
@pytest.mark.parametrize("chans", [(16, 16), (32, 16), (32, 32)])
def test_image_gradient_of_the_strided_convolution(strides, chans):
    images, filters, defv, bp, _ = make_case(53, 2, 11, 13, 7, *chans, (3, 3, 3), 24, np.float32)
    images, filters = _round(images), _round(filters * 0.3)
    want = oracle.sparse_conv3d_fwd(images, filters, defv, bp, strides=strides, dtype=np.float32)
    og = _round(np.random.default_rng(54).uniform(-1, 1, want.shape))
    ig_w, _, _ = oracle.sparse_conv3d_bwd(images, filters, defv, bp, og, strides=strides, dtype=np.float32)
    ig, _, _ = ops.sparse_conv3d_backward(_t(images, bf), _t(filters, bf), float(defv), _t(bp), _t(og, bf), strides)
    assert helpers.rel_err(ig.float().cpu().numpy(), ig_w) <= 1e-2
    assert _lib.lib().chop_umma_timeouts() == 0

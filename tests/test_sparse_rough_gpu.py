"""What base planes cost that are no depth map (random ones) in the convolutions that stage windows of planes: the same work as smooth
ones, in more steps, and no more than a small multiple of their time."""
import numpy as np
import pytest
import torch

from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops

pytestmark = pytest.mark.gpu


def _us(f):
    """Best of five batches of ten calls."""
    best = 1e9
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 100)
    return best


def _bases(H, W):
    r, c = np.indices((H, W))
    smooth = np.round(30 + 20 * np.sin(2 * np.pi * (r / H + 0.3)) * np.cos(2 * np.pi * c / W)).astype(np.int32)
    rough = np.random.default_rng(0).integers(0, 2000, (H, W)).astype(np.int32)
    return [torch.from_numpy(b[None, :, :, None].copy()).cuda() for b in (smooth, rough)]


@pytest.mark.parametrize("chans", [(16, 16), (8, 8), (32, 32)])
def test_stride_1_on_random_base_planes(chans):
    """256x320x9, bfloat16, smooth and random: 36, 59 us (16 -> 16), 33, 49 (8 -> 8), 84, 176 (32 -> 32)."""
    H, W, D = 256, 320, 9
    x = torch.randn((1, H, W, D, chans[0]), device="cuda").bfloat16()
    f = torch.randn((3, 3, 3) + chans, device="cuda").bfloat16()
    z = torch.zeros((), device="cuda", dtype=x.dtype)
    smooth, rough = (_us(lambda: ops.sparse_conv3d_forward(x, f, z, b)) for b in _bases(H, W))
    assert rough <= (2.5 if chans[0] == 32 else 2.0) * smooth, (smooth, rough)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strides", [(2, 2, 2), (2, 2, 1)])
def test_transposed_on_random_base_planes(strides, dtype):
    """256x320x9, 16 <- 16 channels, smooth and random: bfloat16 35, 55 and 32, 51 us, float32 77, 163 and 83, 155."""
    H, W, D = 256, 320, 9
    x = torch.randn([1] + [-(-n // s) for n, s in zip((H, W, D), strides)] + [16], device="cuda").to(dtype)
    f = torch.randn((3, 3, 3, 16, 16), device="cuda").to(dtype)
    z = torch.zeros((), device="cuda", dtype=dtype)
    smooth, rough = (_us(lambda: ops.sparse_conv3d_transpose_forward(x, f, z, b, (H, W, D), strides)) for b in _bases(H, W))
    assert rough <= 3.0 * smooth, (smooth, rough)


@pytest.mark.parametrize("shape,dtype", [((800, 804, 3), torch.bfloat16), ((500, 640, 3), torch.float32)])
@pytest.mark.parametrize("strides", [(2, 2, 2), (2, 2, 1)])
def test_rough_tiles_beyond_the_64th_of_a_cta(shape, dtype, strides):
    """Rough tiles are remembered in 64 bits a CTA, the last of which stands for all that follow: all tiles rough, and only some of
    them, against the kernels that gather tap by tap."""
    H, W, D = shape
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn([1] + [-(-n // s) for n, s in zip(shape, strides)] + [16], generator=g, device="cuda").to(dtype)
    f = (torch.randn((3, 3, 3, 8 if dtype == torch.bfloat16 else 16, 16), generator=g, device="cuda") * 0.25).to(dtype)
    smooth, rough = _bases(H, W)
    mixed = torch.where(torch.rand(smooth.shape, generator=g, device="cuda") < 0.01, rough, smooth)
    knob = "umma_rows" if dtype == torch.bfloat16 else "tile"
    for b in (rough % 61, mixed):
        got = ops.sparse_conv3d_transpose_forward(x, f, 0.5, b, shape, strides)
        _lib.set_tuning(knob, 2)
        try:
            want = ops.sparse_conv3d_transpose_forward(x, f, 0.5, b, shape, strides)
        finally:
            _lib.set_tuning(knob, 1)
        scale = want.abs().max().float()
        # results rounded to bfloat16; float32: some units of 2^-24 times the root of the number of terms
        assert ((got.float() - want.float()).abs().max() <= (2.0 ** -7 if dtype == torch.bfloat16 else 3e-6) * scale).item()
    assert _lib.lib().chop_umma_timeouts() == 0

"""The convolutions that stage windows of planes, at sizes where every CTA takes many tiles: all channel pairs of the bfloat16 stride-1
form, the float32 stride-1 and transposed forms, base planes and values that change from one tile to the next.  Against the kernels
with a thread per output."""
import numpy as np
import pytest
import torch

from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops

pytestmark = pytest.mark.gpu
CHANNELS = (8, 16, 32)


def _bases(kind, B, H, W, slack, seed=0):
    """smooth: one window a tile.  passes: up to one plane more than a window holds.  mixed: smooth, with rough patches."""
    rng = np.random.default_rng(seed)
    r, c = np.indices((H, W))
    smooth = np.round(30 + 20 * np.sin(2 * np.pi * (r / H + 0.3)) * np.cos(2 * np.pi * c / W)).astype(np.int64)
    if kind == "passes":
        smooth = smooth * 0 + rng.integers(0, slack + 2, (H, W))
    if kind == "mixed":
        patch = np.kron(rng.random((H // 7 + 1, W // 11 + 1)) < 0.2, np.ones((7, 11), bool))[:H, :W]
        smooth = np.where(patch, rng.integers(-40, 2000, (H, W)), smooth)
    return torch.from_numpy(np.broadcast_to(smooth[None, :, :, None], (B, H, W, 1)).astype(np.int32).copy()).cuda()


def _both(run):
    """run() with the default kernels, and with a thread per output."""
    got = run()
    for knob in ("umma", "tile"):
        _lib.set_tuning(knob, 0)
    try:
        want = run()
    finally:
        for knob in ("umma", "tile"):
            _lib.set_tuning(knob, 1)
    assert _lib.lib().chop_umma_timeouts() == 0
    return list(zip(got, want))


def _compare(got, want, taps):
    """Both sides round sums of `taps` products: float32 in 24 bits at every addition, 2^-24 of the largest partial sum each (which the
    largest result stands for), results in bfloat16 to one unit in the last place of eight bits apart."""
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
    ok = torch.isfinite(want)
    g, w = got[ok].double(), want[ok].double()
    if got.dtype == torch.bfloat16:
        bound = 2.0 ** -7 * w.abs() + taps * 2.0 ** -24 * w.abs().max()
    else:
        bound = 3e-6 * w.abs().max()          # the root of the number of terms, some units of 2^-24
    assert w.numel() > 0 and bool(((g - w).abs() <= bound).all()), float(((g - w).abs() / bound).max())


@pytest.mark.parametrize("D,kind", [(9, "passes"), (9, "mixed"), (17, "passes"), (17, "mixed")])
@pytest.mark.parametrize("cout", CHANNELS)
@pytest.mark.parametrize("cin", CHANNELS)
def test_bfloat16_stride_1_all_channel_pairs(cin, cout, D, kind):
    B, H, W = (1, 141, 163) if D == 9 else (2, 67, 83)        # 3 to 20 tiles a CTA, none of which divides the image
    g = torch.Generator(device="cuda").manual_seed(cin + cout + D)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()
    images, filters, og = rnd(B, H, W, D, cin), rnd(3, 3, 3, cin, cout) * 0.25, rnd(B, H, W, D, cout)
    bp = _bases(kind, B, H, W, (16 if D <= 10 else 32) - 2 - D)
    run = lambda: (ops.sparse_conv3d_forward(images, filters, 0.75, bp), ops.sparse_conv3d_backward(images, filters, 0.75, bp, og)[0])
    for (got, want), k in zip(_both(run), (cin, cout)):
        _compare(got, want, 27 * k)


def _spoil(x, g):
    """Tiles that float32 computes without pieces between tiles in pieces: blocks of pixels of values near 2^-110, single voxels that are
    no numbers."""
    B, H, W, D, C = x.shape
    block = torch.rand((B, H // 9 + 1, W // 23 + 1), generator=g, device="cuda") < 0.25
    block = block.repeat_interleave(9, 1).repeat_interleave(23, 2)[:, :H, :W]
    x = torch.where(block[..., None, None], x * 2.0 ** -110, x)
    for i, v in enumerate((float("inf"), float("-inf"), float("nan"))):
        at = torch.randint(0, B * H * W * D, (12,), generator=g, device="cuda")
        x.view(-1, C)[at, i] = v
    return x


@pytest.mark.parametrize("values", ["ordinary", "spoilt"])
@pytest.mark.parametrize("kind", ["smooth", "mixed"])
@pytest.mark.parametrize("D", [7, 13])
@pytest.mark.parametrize("chans", [(16, 16), (16, 32), (32, 16), (8, 8)])
def test_float32_stride_1(chans, D, kind, values):
    cin, cout = chans
    B, H, W = 1, 101, 163                                     # 7 and more tiles a CTA
    g = torch.Generator(device="cuda").manual_seed(cin + cout + D)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    images, filters, og = rnd(B, H, W, D, cin), rnd(3, 3, 3, cin, cout), rnd(B, H, W, D, cout)
    if values == "spoilt":
        images, og = _spoil(images, g), _spoil(og, g)
    bp = _bases(kind, B, H, W, 0)

    def run():                                                # the backward's gather form with no padding, and with one
        return (ops.sparse_conv3d_forward(images, filters, 0.75, bp), ops.sparse_conv3d_backward(images, filters, 0.75, bp, og)[0],
                ops.sparse_conv3d_transpose_forward(og, filters, 0.75, bp, (H, W, D)))
    for (got, want), k in zip(_both(run), (cin, cout, cout)):
        _compare(got, want, 27 * k)


@pytest.mark.parametrize("values", ["ordinary", "spoilt"])
@pytest.mark.parametrize("kind", ["smooth", "mixed"])
@pytest.mark.parametrize("strides,chans", [((2, 2, 2), (8, 8)), ((2, 2, 2), (8, 16)), ((2, 2, 2), (16, 8)), ((2, 2, 2), (16, 16)),
                                           ((2, 2, 1), (16, 16))])
def test_float32_transposed(strides, chans, kind, values):
    cin, cout = chans                                         # produced, gathered
    H, W, D = 129, 163, 9                                     # 7 and more tiles a CTA
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    coarse = [-(-n // s) for n, s in zip((H, W, D), strides)]
    images, filters, fine = rnd(1, *coarse, cout), rnd(3, 3, 3, cin, cout), rnd(1, H, W, D, cin)
    if values == "spoilt":
        images = _spoil(images, g)
    bp = _bases(kind, 1, H, W, 0)
    run = lambda: (ops.sparse_conv3d_transpose_forward(images, filters, 0.75, bp, (H, W, D), strides),
                   ops.sparse_conv3d_backward(fine, filters, 0.75, bp, images, strides)[0])
    for got, want in _both(run):
        _compare(got, want, 27 * cout)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strides", [(2, 2, 2), (2, 2, 1)])
@pytest.mark.parametrize("size,D", [((60, 99), 3), ((60, 99), 8), ((60, 99), 9), ((60, 101), 8), ((183, 184), 3), ((185, 184), 3), ((185, 184), 4),
                                    ((185, 184), 5), ((185, 184), 6)])
@pytest.mark.parametrize("chans", [(8, 8), (8, 16), (16, 8), (16, 16), (16, 32)])
def test_transposed_around_the_choice_of_kernel(dtype, strides, size, D, chans):
    """Few planes, on both sides of the image sizes from which the gather per tap takes over."""
    cin, cout = chans
    H, W = size
    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)
    images, filters = rnd(1, *(-(-n // s) for n, s in zip((H, W, D), strides)), cout), rnd(3, 3, 3, cin, cout) * 0.25
    bp = _bases("mixed", 1, H, W, 0)
    run = lambda: (ops.sparse_conv3d_transpose_forward(images, filters, 0.75, bp, (H, W, D), strides),)
    for got, want in _both(run):
        _compare(got, want, 27 * cout)

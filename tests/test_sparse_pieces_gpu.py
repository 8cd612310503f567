"""float32 convolutions in three bfloat16 pieces: values whose pieces or their products would overflow or fall below the normal range
give what float32 multiply-adds give."""
import numpy as np
import pytest
import torch

from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops

pytestmark = pytest.mark.gpu

# op, strides, gathered channels, produced channels: every form that has a kernel in pieces
FORMS = [("conv", (1, 1, 1), 16, 16), ("conv", (1, 1, 1), 16, 32), ("up", (1, 1, 1), 16, 16), ("up", (1, 1, 1), 16, 32),
         ("up", (2, 2, 2), 16, 16), ("up", (2, 2, 2), 8, 8), ("up", (2, 2, 2), 16, 8), ("up", (2, 2, 2), 8, 16), ("up", (2, 2, 1), 16, 16)]
SIZE = (9, 38, 7)


def _run(form, x, w):
    """x [values of a row of voxels], w [weights of the centre tap, gathered x produced]: outputs [voxel, produced]."""
    op, strides, K, N = form
    H, W, D = SIZE
    f = np.zeros((3, 3, 3, K, N) if op == "conv" else (3, 3, 3, N, K), np.float32)
    f[1, 1, 1] = w if op == "conv" else w.T
    coarse = [-(-n // s) for n, s in zip(SIZE, strides)] if op == "up" else SIZE
    images = np.zeros((1, *coarse, K), np.float32)
    images[0, 2, :len(x), 1] = x
    cuda = lambda a: torch.from_numpy(a).cuda()
    bp = torch.zeros((1, H, W, 1), dtype=torch.int32, device="cuda")
    if op == "conv":
        return ops.sparse_conv3d_forward(cuda(images), cuda(f), 0.0, bp).cpu().numpy()[0, 2, :len(x), 1]
    out = ops.sparse_conv3d_transpose_forward(cuda(images), cuda(f), 0.0, bp, SIZE, strides).cpu().numpy()[0]
    return out[2 * strides[0], 0:len(x) * strides[1]:strides[1], strides[2]]


@pytest.mark.parametrize("form", FORMS)
def test_single_products_at_the_ends_of_the_range(form):
    K, N = form[2:]
    big, up = np.float32(2.0 ** 100), np.float32(1.9999 * 2.0 ** 27)
    for x, w in [(big, up), (1e30, 1e12), (-1e30, 1e12), (1.2345e30, 1.3579e12), (3.3e38, 1.0), (1.0, 3.4e38), (2.0 ** -20, 3.4e38),
                 (3.3e38, 1e-37), (1.2345e-13, 1.3579e-13), (1.2345e-30, 1.3579), (1.3579, 1.2345e-31), (1.3579e-19, 1.2345e-19), (0.0, 1e30)]:
        x, w = np.float32(x), np.float32(w)
        xs, ws = np.zeros((16, K), np.float32), np.zeros((K, N), np.float32)
        xs[5, 3], ws[3, N - 2] = x, w
        with np.errstate(over="ignore"):
            want = x * w
        got = _run(form, xs, ws)
        # one product: three pieces of 8 bits each leave 2^-24 of it out, the sums of the pieces' products round three times more
        assert got[5, N - 2] == want or abs(got[5, N - 2] - want) <= 4 * 2.0 ** -24 * abs(want), (x, w, got[5, N - 2])
        got[5, N - 2] = 0
        assert np.array_equal(got, np.zeros_like(got)), (x, w)
    assert _lib.lib().chop_umma_timeouts() == 0


@pytest.mark.parametrize("form", FORMS)
def test_sums_that_overflow_have_the_sign_of_their_terms(form):
    K, N = form[2:]
    rng = np.random.default_rng(3)
    xs, ws = (1e30 * rng.uniform(1, 2, (16, K))).astype(np.float32), (1e12 * rng.uniform(1, 2, (K, N))).astype(np.float32)
    ws[:, 1] *= -1
    got = _run(form, xs, ws)
    assert (got[:, 1] == -np.inf).all() and (np.delete(got, 1, 1) == np.inf).all()
    got = _run(form, xs, ws * np.float32(2.0 ** -40))      # the same sums below the end of the range
    want = xs.astype(np.float64) @ (ws * np.float32(2.0 ** -40)).astype(np.float64)
    assert np.abs(got / want - 1).max() <= K * 2.0 ** -24


@pytest.mark.parametrize("form", FORMS)
def test_small_values_beside_ordinary_ones(form):
    """A step is computed in pieces if its largest value allows it; what its small values lose is below 2^-133 of a value, the step of
    bfloat16's subnormal numbers."""
    K, N = form[2:]
    rng = np.random.default_rng(4)
    xs = rng.standard_normal((16, K)).astype(np.float32)
    ws = rng.standard_normal((K, N)).astype(np.float32)
    xs[3:] *= np.exp2(-100.0 - 2 * np.arange(13))[:, None].astype(np.float32)   # 2^-100 .. 2^-124 beside three ordinary voxels
    got = _run(form, xs, ws).astype(np.float64)
    want = xs.astype(np.float64) @ ws.astype(np.float64)
    terms = np.abs(xs).astype(np.float64) @ np.abs(ws).astype(np.float64)
    # and products below 2^-126 that the tensor core may round to a multiple of 2^-149: K of them and their sums
    bound = K * 2.0 ** -24 * terms + 2.0 ** -133 * np.abs(ws).astype(np.float64).sum(0) + 8 * K * 2.0 ** -149
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max(1)


@pytest.mark.parametrize("spread", [3, 60])       # base planes that fit a window, and that do not
@pytest.mark.parametrize("default", [0.0, 0.75])
@pytest.mark.parametrize("form", FORMS)
def test_values_that_are_no_numbers(form, default, spread):
    """Infinities and NaN in either operand, against the kernels with a thread per output: where results are not finite, and the rest.
    A tap that is padding multiplies the default value in the forward forms, also a zero, and adds nothing in the gradients."""
    op, strides, K, N = form
    H, W, D = SIZE
    rng = np.random.default_rng(spread)
    rnd = lambda *s: rng.standard_normal(s).astype(np.float32)
    coarse = [-(-n // s) for n, s in zip(SIZE, strides)]
    images, filters = rnd(1, *coarse, K), rnd(*((3, 3, 3, K, N) if op == "conv" else (3, 3, 3, N, K)))
    bp = torch.from_numpy(rng.integers(0, spread + 1, (1, H, W, 1)).astype(np.int32)).cuda()
    fine = torch.zeros((1, H, W, D, N), device="cuda")
    bad_images, bad_filters, tiny = images.copy(), filters.copy(), images.copy()
    for a, at in ((bad_images, (0, 2, 3, 1)), (bad_filters, (0, 2, 1))):
        a[at + (3,) * (5 - len(at))] = np.inf
        a[(0, 1, 2, 2, 5)[:len(a.shape)] if a is bad_images else (2, 0, 1, 5, 4)] = np.nan
    tiny *= np.float32(2.0 ** -110)               # a step of these is computed without pieces
    tiny[0, :, 10:] = images[0, :, 10:]           # beside steps that are not

    def run(i, f):
        i, f = torch.from_numpy(i).cuda(), torch.from_numpy(f).cuda()
        if op == "conv":
            return [ops.sparse_conv3d_forward(i, f, default, bp, strides).cpu().numpy()]
        return [ops.sparse_conv3d_transpose_forward(i, f, default, bp, SIZE, strides).cpu().numpy(),
                ops.sparse_conv3d_backward(fine, f, default, bp, i, strides)[0].cpu().numpy()]

    for i, f in ((bad_images, filters), (images, bad_filters), (tiny, filters)):
        got = run(i, f)
        _lib.set_tuning("tile", 0)
        try:
            want = run(i, f)
        finally:
            _lib.set_tuning("tile", 1)
        for g, w in zip(got, want):
            assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isposinf(g), np.isposinf(w))
            assert np.array_equal(np.isneginf(g), np.isneginf(w))
            ok = np.isfinite(w)
            assert np.isfinite(w).any() and (np.abs(g[ok] - w[ok]) <= 3e-6 * np.abs(w[ok]).max()).all()
            if i is tiny and default == 0.0:      # and the voxels that see small values alone, relative to themselves
                small = np.abs(w) < 2.0 ** -90
                assert small.any() and (np.abs(g[small] - w[small]) <= 3e-6 * np.abs(w[small]).max()).all()

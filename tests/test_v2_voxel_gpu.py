"""CostVolumeV2 forward with eight channels (a lane per voxel): both types, MEAN and MIN, groups of one, two and four channels, depth
counts around the planes of a warp, ragged pixel counts, views that miss part of the volume, depth ranges, against the oracle and,
for MIN, bit for bit.  The gradient's blocks of two and four planes on the same cases."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import synth
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G", [8, 4, 2])
@pytest.mark.parametrize("shape", [(1, 1, 3, 5, 1), (2, 3, 9, 11, 4), (1, 2, 7, 13, 9), (3, 4, 5, 31, 16), (1, 5, 12, 10, 19), (1, 2, 2, 3, 20)])
@pytest.mark.parametrize("reduce", ["MEAN", "MIN"])
def test_forward_and_gradient(dtype, G, shape, reduce):
    B, N, H, W, D = shape
    c = helpers.make_case(2, 90 + G, B, N, H, W, 8, D, "random" if H > 7 else "rot_y", np.float32)
    t = {k: torch.from_numpy(c[k]).to(dtype) for k in ("ref", "src")}
    f = {k: t[k].float().numpy() for k in t}
    want, mask = oracle.cost_fwd(2, f["ref"], f["src"], c["depth"], None, c["Rs"], c["Ts"], reduce, G, True, np.float32)
    args = [t["ref"].cuda(), t["src"].cuda(), torch.from_numpy(c["depth"]).cuda(), None, torch.from_numpy(c["Rs"]).cuda(),
            torch.from_numpy(c["Ts"]).cuda()]
    got, m = ops.cost_forward(2, *args, reduce, G)
    assert np.array_equal(m.cpu().numpy().reshape(mask.shape), mask)
    if reduce == "MIN":
        assert np.array_equal(got.cpu().numpy().reshape(want.shape), want)
    else:
        assert helpers.rel_err(got.cpu().numpy().reshape(want.shape), want) <= 1e-5
    if D > 2:   # a depth range leaves the other planes alone
        out = (torch.full_like(got, 7.0), torch.full_like(m, 7))
        ops.cost_forward(2, *args, reduce, G, d_range=(1, D - 1), out=out)
        assert torch.equal(out[0][..., 1:D - 1, :], got[..., 1:D - 1, :]) and torch.equal(out[1][..., 1:D - 1, :], m[..., 1:D - 1, :])
        assert bool((out[0][..., [0, D - 1], :] == 7).all()) and bool((out[1][..., [0, D - 1], :] == 7).all())
    cg = np.random.default_rng(3).standard_normal(want.shape).astype(np.float32)
    grads = ops.cost_backward(2, *args, torch.from_numpy(cg).cuda(), m, reduce, G)
    want_g = oracle.cost_bwd(2, f["ref"], f["src"], c["depth"], None, c["Rs"], c["Ts"], cg, mask, reduce, G, True, np.float32)
    for g, w in zip(grads, want_g):
        assert helpers.rel_err(g.cpu().numpy().reshape(w.shape), w) <= 1e-4


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G", [8, 2])
@pytest.mark.parametrize("N,D", [(1, 8), (1, 16), (1, 18), (2, 17), (2, 18), (2, 34), (3, 16), (3, 18), (3, 19), (3, 32), (4, 24)])   # both sides of
                         # the choice of kernel and of planes
@pytest.mark.parametrize("reduce", ["MEAN", "MIN"])
@pytest.mark.parametrize("shift", [0, 16])   # bytes by which the features miss a 32-byte boundary
def test_choice_of_kernel(dtype, G, N, D, reduce, shift):
    c = helpers.make_case(2, 17, 1, N, 6, 9, 8, D, "random", np.float32)
    t = {k: torch.from_numpy(c[k]).to(dtype) for k in ("ref", "src")}
    f = {k: t[k].float().numpy() for k in t}
    want, mask = oracle.cost_fwd(2, f["ref"], f["src"], c["depth"], None, c["Rs"], c["Ts"], reduce, G, True, np.float32)

    def place(x):
        room = torch.empty(x.numel() + 32, dtype=x.dtype, device="cuda")
        n = shift // x.element_size()
        return room[n:n + x.numel()].view(x.shape).copy_(x)

    cuda = lambda k: torch.from_numpy(c[k]).cuda()
    ref, src = place(t["ref"]), place(t["src"])
    assert ref.data_ptr() % 32 == shift
    got, m = ops.cost_forward(2, ref, src, cuda("depth"), None, cuda("Rs"), cuda("Ts"), reduce, G)
    assert np.array_equal(m.cpu().numpy().reshape(mask.shape), mask)
    if reduce == "MIN":
        assert np.array_equal(got.cpu().numpy().reshape(want.shape), want)
    else:
        assert helpers.rel_err(got.cpu().numpy().reshape(want.shape), want) <= 1e-5


@pytest.mark.parametrize("G", [8, 4])
def test_features_larger_than_l2(G):
    """Source features of more than 126 MB are read in 32-byte loads where their addresses allow it, otherwise as smaller ones are."""
    N, H, W, D = 4, 1000, 1100, 4
    g = torch.Generator(device="cuda").manual_seed(G)
    Rs, Ts = (torch.from_numpy(x).to("cuda", torch.float32) for x in synth.random_cameras(np.random.default_rng(1), 1, N, H, W))
    depth = 600.0 + 200.0 * torch.rand((1, H, W, D), generator=g, device="cuda")
    room = torch.randn((N + 1) * H * W * 8 + 8, generator=g, device="cuda")

    def run(shift):
        x = torch.empty_like(room)
        x[shift:shift + room.numel() - 8] = room[:-8]
        ref = x[shift:shift + H * W * 8].view(1, H, W, 8)
        src = x[shift + H * W * 8:shift + room.numel() - 8].view(1, N, H, W, 8)
        assert src.data_ptr() % 32 == shift * 4
        return ops.cost_forward(2, ref, src, depth, None, Rs, Ts, "MEAN", G)

    (a, ma), (b, mb) = run(0), run(4)
    assert torch.equal(ma, mb) and int(ma.max()) == N and torch.equal(a, b)

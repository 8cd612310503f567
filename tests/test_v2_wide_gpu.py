"""The eight-channels-per-lane CostVolumeV2 forward (bfloat16) at every channel / group pair that takes it: depth counts
around its block of planes, ragged pixel counts, views that miss part of the volume, a depth range, against the oracle on the
rounded features and against the four-channel kernel (knob "packed" off)."""
import numpy as np
import pytest
import torch

import oracle
from custom_helper_op_b200 import _lib
from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,G", [(8, 8), (8, 4), (8, 2), (16, 16), (16, 8), (32, 32)])
@pytest.mark.parametrize("shape", [(1, 1, 3, 5, 1), (2, 3, 9, 11, 4), (1, 2, 7, 13, 9), (1, 5, 12, 10, 21)])
@pytest.mark.parametrize("camera", ["random", "rot_y"])
def test_wide_forward(C, G, shape, camera):
    B, N, H, W, D = shape
    c = helpers.make_case(2, 70 + C + G, B, N, H, W, C, D, camera, np.float32)
    bf = {k: torch.from_numpy(c[k]).to(torch.bfloat16) for k in ("ref", "src")}
    want, mask = oracle.cost_fwd(2, bf["ref"].float().numpy(), bf["src"].float().numpy(), c["depth"], None, c["Rs"], c["Ts"],
                                 "MEAN", G, True, np.float32)
    args = [bf["ref"].cuda(), bf["src"].cuda(), torch.from_numpy(c["depth"]).cuda(), None, torch.from_numpy(c["Rs"]).cuda(),
            torch.from_numpy(c["Ts"]).cuda(), "MEAN", G]
    got, m = ops.cost_forward(2, *args)
    assert np.array_equal(m.cpu().numpy().reshape(mask.shape), mask)
    assert helpers.rel_err(got.cpu().numpy().reshape(want.shape), want) <= 1e-5
    try:
        _lib.set_tuning("packed", 0)
        old, _ = ops.cost_forward(2, *args)
    finally:
        _lib.set_tuning("packed", 1)
    assert helpers.rel_err(got.cpu().numpy(), old.cpu().numpy()) <= 2e-6
    if D > 2:   # a depth range leaves the other planes alone
        out = (torch.full_like(got, 7.0), torch.full_like(m, 7))
        ops.cost_forward(2, *args, d_range=(1, D - 1), out=out)
        assert torch.equal(out[0][..., 1:D - 1, :], got[..., 1:D - 1, :]) and torch.equal(out[1][..., 1:D - 1, :], m[..., 1:D - 1, :])
        assert bool((out[0][..., [0, D - 1], :] == 7).all()) and bool((out[1][..., [0, D - 1], :] == 7).all())

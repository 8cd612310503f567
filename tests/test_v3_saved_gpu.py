"""CostVolumeV3 MEAN: the gradient that uses the winners recorded by the forward pass, against the oracle."""
import numpy as np
import pytest
import torch

from custom_helper_op_b200.python.ops import custom_helper_ops as ops
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,groups", [(8, 2), (16, 4), (32, 8), (16, 2), (32, 4)])
@pytest.mark.parametrize("N,D", [(1, 1), (3, 8), (2, 21)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_recorded_winners(C, groups, N, D, dtype):
    c = helpers.make_case(4, 71, 2, N, 5, 7, C, D, "random", np.float32)   # 70 pixels: a ragged last warp
    for k in ("ref", "src"):
        c[k] = torch.from_numpy(c[k]).to(dtype).float().numpy()
    want = helpers.oracle_fwd_bwd(4, c, "MEAN", groups, True, np.float32)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to("cuda:0") for k, v in c.items()}
    ref, src = (t[k].to(dtype).requires_grad_(True) for k in ("ref", "src"))
    base = t["depth"].requires_grad_(True)
    cost, mask = ops.cost_volume_v3(ref, src, base, t["offsets"], t["Rs"], t["Ts"], "MEAN", groups)
    assert helpers.bits_equal(mask.cpu().numpy(), want["mask"])
    assert helpers.bits_equal(cost.detach().cpu().numpy(), want["cost"])
    got = torch.autograd.grad(cost, (ref, src, base), torch.from_numpy(want["cost_grad"]).to("cuda:0"))
    tol = 1e-4 if dtype == torch.float32 else 1e-2
    for a, b in zip(got, (want["ref_grad"], want["src_grad"], want["depth_grad"])):
        assert helpers.rel_err(a.float().cpu().numpy().reshape(b.shape), b) <= tol

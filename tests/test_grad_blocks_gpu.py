"""CostVolume and CostAggregate gradients with eight and sixteen channels around the choice between blocks of two and four, or four and eight
planes: depth counts that one divides and the other does not, chunks that end inside a block, against the oracle."""
import numpy as np
import pytest

from custom_helper_op_b200 import _lib
from tests import helpers
from tests.test_cost_volume_gpu import check, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,reduce", [(1, "MEAN"), (3, "MEAN"), (3, "MIN")])
@pytest.mark.parametrize("C", [8, 16])
@pytest.mark.parametrize("N", [1, 2, 4])
@pytest.mark.parametrize("D", [16, 17, 20, 23, 33, 45])
def test_against_the_oracle(kind, reduce, C, N, D):
    c = helpers.make_case(kind, 100 * N + D, 1, N, 7, 11, C, D, "random", np.float32)
    want = helpers.oracle_fwd_bwd(kind, c, reduce, 1, True, np.float32)
    for chunk in (0, 12, 64):                 # planes of a work item: the host's choice, blocks inside it, all planes
        _lib.set_tuning("bwd_chunk", chunk)
        try:
            got = run_gpu(kind, c, reduce, 1, True, want["cost_grad"])
        finally:
            _lib.set_tuning("bwd_chunk", 0)
        check(got, want, np.float32, exact_cost=reduce == "MIN")

"""float32 gradients rounded to bfloat16 two buffers at a time: remainders, unequal sizes, misaligned buffers, specials."""
import ctypes

import pytest
import torch

from custom_helper_op_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0,n1,shift", [(1, 0, 0), (7, 8, 0), (9, 4099, 0), (4096, 1, 0), (300001, 77, 0), (64, 65, 1)])
def test_narrow(n0, n1, shift):
    g = torch.Generator(device="cuda").manual_seed(n0)
    src = [torch.randn(n + shift, generator=g, device="cuda")[shift:] for n in (n0, n1)]
    src[0][0] = float("inf")
    src[0][-1] = 1.00390625   # halfway between two bfloat16 values
    dst = [torch.full((n + shift + 8,), 7.0, dtype=torch.bfloat16, device="cuda") for n in (n0, n1)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    f = _lib.lib().chop_narrow_bf16
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64] * 2 + [ctypes.c_void_p]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert f(p(src[0]), p(dst[0][shift:]), n0, p(src[1]) if n1 else None, p(dst[1][shift:]) if n1 else None, n1, stream) == 0
    for s, d, n in zip(src, dst, (n0, n1)):
        assert torch.equal(d[shift:shift + n], s.to(torch.bfloat16))
        assert bool((d[shift + n:] == 7.0).all()) and bool((d[:shift] == 7.0).all())

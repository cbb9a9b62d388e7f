"""gnb200_cast_params: fp32 parameters rounded to a 16-bit type in one launch, as torch rounds them."""
import ctypes

import pytest
import torch


def _raw():
    from channels_last_groupnorm_b200 import _native as nt

    f = nt.lib.gnb200_cast_params
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    return f


def test_argument_checks():
    f = _raw()
    one = 64  # validation fails before anything is launched
    assert f(one, one, 8, 0, one, one, None) == -1  # fp32 is no 16-bit type
    assert f(one, one, 0, 1, one, one, None) == -1
    assert f(None, one, 8, 1, one, one, None) == -1 and f(one, one, 8, 2, one, None, None) == -1


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,code", [(torch.float16, 1), (torch.bfloat16, 2)], ids=["fp16", "bf16"])
@pytest.mark.parametrize("C", [1, 7, 255, 256, 257, 2048])
def test_rounding(C, dtype, code):
    torch.manual_seed(C)
    w, b = torch.randn(2, C, device="cuda").mul(100.0).unbind(0)
    w[0] = float("inf")
    b[0] = 1e-7  # subnormal in fp16
    wo, bo = (torch.zeros(C + 1, device="cuda", dtype=dtype) for _ in range(2))
    assert _raw()(w.data_ptr(), b.data_ptr(), C, code, wo.data_ptr(), bo.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(wo[:C], w.to(dtype)) and torch.equal(bo[:C], b.to(dtype)) and wo[C] == 0 and bo[C] == 0

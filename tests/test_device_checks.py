"""Calls that are refused before anything is launched, seen without a GPU: fake tensors of two devices."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="host checks: their operands are no memory of a GPU")


def _fake(*shape, device=0, dtype=torch.float16):
    with FakeTensorMode(allow_non_fake_inputs=True):
        return torch.empty(*shape, device=f"cuda:{device}", dtype=dtype)


def test_conv_of_two_devices(built_lib):
    import flash_dropout.functional as F
    with pytest.raises(RuntimeError, match="same device"):
        F.cuda_blockwise_dropout_conv2d(_fake(1, 8, 8, 8), _fake(8, 8, 3, 3, device=1), 128, 0.5)


def test_plan_of_another_device(built_lib):
    import types
    import flash_dropout.functional as F
    plan = types.SimpleNamespace(buf=_fake(4096, device=1, dtype=torch.uint8), R=1, C=1, origin=None)
    with pytest.raises(RuntimeError, match="plan must be on the device"):
        F.cuda_blockwise_dropout_matmul(_fake(128, 128), _fake(128, 128), 128, 0.5, plan=plan)
    with pytest.raises(RuntimeError, match="plan must be on the device"):
        F.cuda_blockwise_dropout_conv2d(_fake(1, 8, 8, 8), _fake(8, 8, 3, 3), 128, 0.5, padding=(1, 1), plan=plan)


def test_mask_of_another_device(built_lib):
    from flash_dropout.cuda.binding_gemm import GEMM
    mask = _fake(1, 1, device=1, dtype=torch.bool)
    for call in (GEMM().gemm_dsd, GEMM().gemm_sdd):
        with pytest.raises(RuntimeError, match="Mask must be on the operands' device"):
            call(_fake(128, 128), _fake(128, 128), mask, 128, 2.0)


def test_weight_copy_of_another_device(built_lib):
    import flash_dropout.functional as F
    f32 = dict(dtype=torch.float32)
    torch.set_autocast_enabled("cuda", True)         # (torch.autocast turns itself off where there is no GPU)
    torch.set_autocast_dtype("cuda", torch.float16)
    try:
        with pytest.raises(RuntimeError, match="same device"):
            F.cuda_blockwise_dropout_matmul(_fake(128, 128, **f32), _fake(128, 128, **f32), 128, 0.5,
                                            wgrad=(_fake(128, 128, **f32), False, None), weight_lowp=_fake(128, 128, device=1))
    finally:
        torch.set_autocast_enabled("cuda", False)

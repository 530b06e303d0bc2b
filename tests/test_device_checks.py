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

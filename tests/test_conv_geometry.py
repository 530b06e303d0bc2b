"""A filter that does not fit the padded input is refused before anything is launched, whatever the stride."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="host checks: their operands are no memory of a GPU")

# H, W, R, S, padding, stride: larger than the input by less than the stride
TOO_LARGE = [(2, 8, 3, 3, (0, 1), (2, 1)), (8, 2, 3, 3, (1, 0), (1, 2)), (2, 2, 5, 5, (1, 1), (3, 3)), (2, 8, 3, 3, (0, 1), (1, 1))]


@pytest.mark.parametrize("H,W,R,S,pad,stride", TOO_LARGE)
def test_operator(built_lib, H, W, R, S, pad, stride):
    import flash_dropout.functional as F
    with FakeTensorMode(allow_non_fake_inputs=True):
        x = torch.empty(1, 8, H, W, device="cuda:0", dtype=torch.float16)
        k = torch.empty(8, 8, R, S, device="cuda:0", dtype=torch.float16)
    with pytest.raises(RuntimeError, match="does not fit the padded input"):
        F.cuda_blockwise_dropout_conv2d(x, k, 128, 0.5, padding=pad, stride=stride)


@pytest.mark.parametrize("H,W,R,S,pad,stride", TOO_LARGE)
def test_library(built_lib, H, W, R, S, pad, stride):
    """The geometry check comes before the pointers are used: they lead nowhere here."""
    nowhere = 1 << 20
    geom = (1, 8, H, W, R, S, *pad, *stride, 1, 1)
    k64 = -(-8 * R * S // 64) * 64
    assert built_lib.sd_im2col_kept_panels(nowhere, *geom, nowhere, k64, None, None) == -1
    assert b"does not fit" in built_lib.sd_last_error()
    assert built_lib.sd_col2im_kept_panels(nowhere, k64, *geom, nowhere, None, 0, None) == -1
    assert built_lib.sd_conv_fused_supported(*geom) == 0

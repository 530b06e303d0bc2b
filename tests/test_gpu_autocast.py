"""The pieces of a layer under autocast that leave or enter in fp32: the input cast and the input gradient."""
import pytest
import torch

from oracle import masked_dense as md
from oracle import philox_mask as pm

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("na,nb", [(1, 0), (7, 8), (0, 9), (4099, 3 * 1024 * 1024 + 5)])
def test_cast16_rounds_like_torch(built_lib, na, nb, dtype):
    """Bit-exact for lengths around the eight-element step, with either tensor missing."""
    from flash_dropout import _lib
    a, b = torch.randn(max(na, 1), device=DEV), torch.randn(max(nb, 1), device=DEV)
    a16, b16 = (torch.full((t.numel() + 8,), 7.0, device=DEV, dtype=dtype) for t in (a, b))
    _lib.check(built_lib.sd_cast16(a.data_ptr(), a16.data_ptr(), na, b.data_ptr(), b16.data_ptr(), nb, _lib.dtype_code(dtype),
                                   torch.cuda.current_stream().cuda_stream))
    for src, dst, n in ((a, a16, na), (b, b16, nb)):
        assert torch.equal(dst[:n], src[:n].to(dtype)) and bool((dst[n:] == 7.0).all())


@pytest.mark.parametrize("M,N,K,masked", [(128, 128, 128, False), (300, 264, 392, False), (300, 264, 392, True),
                                          (256, 4096, 256, False), (130, 8, 1032, True), (2048, 256, 1024, False)])
def test_input_gradient_in_fp32(built_lib, M, N, K, masked):
    """sd_gemm_sdd_f32 against the oracle: whole tiles, ragged edges, the split schedule (long reduction, few tiles), the
    ReLU mask.  Sums of at most N = 4096 products of fp16 values in fp32: the error bound is N * 2^-24 of the sum of
    magnitudes, below 1e-3 of the O(1) results; unlike a 16-bit result nothing is rounded at the end."""
    from flash_dropout import _lib
    from flash_dropout.cuda import binding_gemm as bg
    p = 0.4
    g = torch.Generator().manual_seed(M + N + K)
    x = (torch.randn(M, K, generator=g) * K ** -0.25).half()
    w = (torch.randn(N, K, generator=g) * K ** -0.25).half()
    dy = (torch.randn(M, N, generator=g) * N ** -0.25).half()
    mask = pm.block_mask(M, K, 128, p, seed=3, offset=1)
    _, want, _ = md.forward_backward(x, mask, 128, p, w, dy)
    if masked:
        want = want * (x > 0)
    plan = bg.BlockPlan.from_mask(torch.from_numpy(mask).to(DEV), M, K, 128)
    xd, wd, dyd = x.to(DEV), w.to(DEV), dy.to(DEV)
    dx = torch.full((M, K), float("nan"), device=DEV)
    _lib.check(built_lib.sd_gemm_sdd_f32(dyd.data_ptr(), N, 1, wd.data_ptr(), 1, K, dx.data_ptr(), K, 1, M, K, N, plan.buf.data_ptr(),
                                         xd.data_ptr() if masked else None, K, 1 / (1 - p), _lib.dtype_code(x.dtype),
                                         bg.workspace(DEV).data_ptr(), bg.status_word(DEV).data_ptr(),
                                         torch.cuda.current_stream().cuda_stream))
    torch.testing.assert_close(dx.cpu(), want.float(), rtol=1e-3, atol=1e-3)


def test_forward_mode_is_refused(built_lib):
    """No forward derivative is implemented: a dual tensor raises instead of losing its tangent."""
    import flash_dropout.functional as F
    import torch.autograd.forward_ad as fwad
    from flash_dropout.layers.norm import layer_norm
    x = torch.randn(128, 128, device=DEV, dtype=torch.float16)
    img = torch.randn(1, 8, 8, 8, device=DEV, dtype=torch.float16)
    with fwad.dual_level():
        for call in (lambda: F.cuda_blockwise_dropout_matmul(fwad.make_dual(x, x), x, 128, 0.5),
                     lambda: F.cuda_blockwise_dropout_conv2d(fwad.make_dual(img, img), torch.randn(8, 8, 3, 3, device=DEV).half(), 128, 0.5),
                     lambda: layer_norm(fwad.make_dual(x.float(), x.float()), (128,), torch.ones(128, device=DEV), None, 1e-5)):
            with pytest.raises(RuntimeError, match="forward AD"):
                call()


def test_errors_in_backward_keep_their_type(built_lib):
    """What the gradient callback raises on autograd's thread is what the caller of backward() catches."""
    import flash_dropout.functional as F
    x = torch.randn(128, 128, device=DEV, dtype=torch.float16, requires_grad=True)

    def notify():
        raise KeyError("bucket")

    y = F.cuda_blockwise_dropout_matmul(x, x.detach(), 128, 0.5, wgrad=(torch.empty(128, 128, device=DEV), False, notify))
    with pytest.raises(KeyError, match="bucket"):
        y.sum().backward()

"""col2im staged through shared memory, and its fp32 result, at the geometries where strips and channel groups end."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")

GEOMS = [  # N, C, H, W, R, S, padding, stride, dilation
    (2, 5, 7, 7, 3, 3, (1, 1), (1, 1), (1, 1)),       # small images: several channels per CTA, the last group short
    (1, 3, 64, 60, 5, 5, (2, 2), (1, 1), (1, 1)),     # runs of one image exceed the budget: several strips, the last one short
    (2, 4, 33, 30, 3, 3, (1, 1), (2, 2), (1, 1)),     # strides that are a power of two, odd height
    (1, 4, 20, 23, 3, 2, (2, 0), (3, 3), (1, 1)),     # strides that are not, input rows no output row reads
    (2, 3, 17, 19, 3, 3, (2, 2), (1, 2), (2, 2)),     # dilated rows and columns
    (2, 3, 18, 21, 3, 3, (1, 1), (2, 2), (1, 1)),     # pairs of results with an odd width: the last pair is cut, single stores
    (1, 3, 56, 70, 5, 5, (2, 2), (2, 2), (1, 1)),     # more pairs than lanes; taps of either parity
    (1, 2, 14, 15, 1, 7, (0, 3), (1, 1), (1, 1)),     # the widest filter the strips take
    (1, 2, 14, 15, 2, 9, (0, 4), (2, 1), (1, 1)),     # one wider: element by element
    (2, 4, 16, 16, 3, 3, (1, 1), (1, 1), (1, 1)),     # the 3x3 kernel with an fp32 result
    (2, 4, 12, 16, 5, 5, (2, 2), (1, 1), (1, 1)),     # the row kernel with an fp32 result
]


@pytest.mark.parametrize("geom", GEOMS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_col2im_against_fold(built_lib, geom, dtype):
    """Against F.fold in fp32 of the masked matrix: the same at most R*S fp32 additions in another order, so the fp32 result
    agrees to R*S * 2^-24 of the sum of magnitudes (< 3e-5 here); the 16-bit result is that one rounded once."""
    from flash_dropout import _lib
    from flash_dropout.cuda.binding_gemm import BlockPlan
    N, C, H, W, R, S, pad, st, dil = geom
    P = (H + 2 * pad[0] - dil[0] * (R - 1) - 1) // st[0] + 1
    Q = (W + 2 * pad[1] - dil[1] * (S - 1) - 1) // st[1] + 1
    M, K = N * P * Q, C * R * S
    Kg, Mp = -(-K // 64) * 64, -(-M // 128) * 128
    g = torch.Generator(device=DEV).manual_seed(K)
    dcol = torch.randn(Kg, Mp, generator=g, device=DEV).to(dtype)
    mask = torch.rand(-(-M // 128), -(-Kg // 128), generator=g, device=DEV) < 0.4
    keep = (~mask).repeat_interleave(128, 0).repeat_interleave(128, 1)[:M, :K].T
    want = TF.fold((dcol[:K, :M].float() * keep).view(K, N, P * Q).permute(1, 0, 2), (H, W), (R, S), padding=pad, stride=st, dilation=dil)
    plan = BlockPlan.from_mask(mask, M, Kg, 128)
    panels = dcol.view(Kg, Mp // 128, 128).permute(1, 0, 2).contiguous()
    for f32 in (True, False):
        dx = torch.full((N, C, H, W), float("nan"), device=DEV, dtype=torch.float32 if f32 else dtype)
        fn = built_lib.sd_col2im_kept_panels_f32 if f32 else built_lib.sd_col2im_kept_panels
        _lib.check(fn(panels.data_ptr(), Kg, N, C, H, W, R, S, *pad, *st, *dil, dx.data_ptr(), plan.buf.data_ptr(),
                      _lib.dtype_code(dtype), torch.cuda.current_stream().cuda_stream))
        if f32:
            torch.testing.assert_close(dx, want, rtol=1e-5, atol=3e-5)
            full = dx
        else:
            assert torch.equal(dx, full.to(dtype))

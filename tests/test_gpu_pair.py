"""The CTA-pair products at the edges of their tiles: slabs and row blocks that hang over, odd numbers of column pairs, kept
tiles left over, row blocks that keep nothing, every operand and result layout, against the masked product in fp64."""
import pytest
import torch

from oracle import masked_dense as md
from oracle import philox_mask as pm

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _operands(M, N, K, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    a = (torch.randn(M, K, generator=g) * K ** -0.25).to(dtype).to(DEV)
    b = (torch.randn(N, K, generator=g) * K ** -0.25).to(dtype).to(DEV)
    return a, b


def _keep(mask, M, N):
    return md._keep_matrix(mask, M, N, 128).to(DEV).double()


def _major(t, col):
    return t.T.contiguous().T if col else t


# sums of O(1) results in fp32, rounded once: half an ulp of the 16-bit type, plus the sums' own error (below 1e-4)
TOL = {torch.float16: 2 ** -11, torch.bfloat16: 2 ** -8}


def _check(got, want, dtype, what):
    err = (got.double() - want).abs()
    bound = TOL[dtype] * want.abs() + 1e-4 if got.dtype != torch.float32 else 1e-4 * want.abs() + 1e-4
    assert bool((err <= bound).all()), f"{what}: {float((err - bound).max())} over the bound"


# entries of the launch per pair: fewer than one wave (all single), a wave and a short rest, several waves; M, N around the
# 128-row block, the 128-row slab and the 256-row pair of slabs; K with a half K tile at the end and kept or not
SHAPES = [(4736, 512, 1024), (2432, 1032, 1096), (2441, 1160, 1272), (8192, 1288, 1024), (9608, 2056, 1160), (4096, 4096, 2048)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_dsd(built_lib, M, N, K, dtype):
    from flash_dropout import _lib
    from flash_dropout.cuda.binding_gemm import BlockPlan, dsd
    a, b = _operands(M, N, K, dtype, M + N + K)
    mask = pm.block_mask(M, K, 128, 0.5, seed=11, offset=M % 7)
    mask[1] = True                                  # a row block that keeps nothing
    mask[2] = True
    mask[2, -1] = False                             # and one that keeps the last, possibly half, K tile only
    plan = BlockPlan.from_mask(torch.from_numpy(mask).to(DEV), M, K, 128)
    want = 2 * (a.double() * _keep(mask, M, K)) @ b.double().T
    for ca in (False, True):
        for cb in (False, True):
            if (ca and M % 8) or (cb and N % 8):
                continue                            # 16-byte rows for the loads
            for cout in (False, True):
                out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
                if cout:
                    out = torch.full((N, (M + 7) // 8 * 8), float("nan"), device=DEV, dtype=dtype)[:, :M].T
                dsd(_major(a, ca), _major(b, cb), plan, _lib.SD_PLAN_ROWS, 2.0, out=out)
                _check(out, want, dtype, f"dsd col-major a={ca} b={cb} out={cout}")
    got = dsd(a, b, plan, _lib.SD_PLAN_ROWS, 2.0, relu=True)
    _check(got, want.clamp(min=0), dtype, "relu")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_sdd(built_lib, M, N, K, dtype):
    """Kept tiles left over in every number, zeros in the dropped ones."""
    from flash_dropout.cuda.binding_gemm import BlockPlan, sdd
    a, b = _operands(M, N, K, dtype, M + 3 * N + K)
    mask = pm.block_mask(M, N, 128, 0.4, seed=12, offset=N % 5)
    for r in range(min(mask.shape[0], mask.shape[1] + 1)):      # 0, 1, 2, ... kept tiles
        mask[r] = True
        mask[r, mask.shape[1] - r:] = False
    plan = BlockPlan.from_mask(torch.from_numpy(mask).to(DEV), M, N, 128)
    keep = _keep(mask, M, N)
    want = 1.5 * (a.double() @ b.double().T) * keep
    for ca in (False, True):
        for cb in (False, True):
            if (ca and M % 8) or (cb and N % 8):
                continue
            got = sdd(_major(a, ca), _major(b, cb), plan, 1.5)
            _check(got, want, dtype, f"sdd col-major a={ca} b={cb}")
            assert bool((got[keep == 0] == 0).all())


@pytest.mark.parametrize("M,N,K", SHAPES[1:5])
def test_fp32_results_and_dense(built_lib, M, N, K):
    from flash_dropout import _lib
    from flash_dropout.cuda.binding_gemm import BlockPlan, GEMM, dsd
    a, b = _operands(M, N, K, torch.float16, M)
    mask = pm.block_mask(M, K, 128, 0.5, seed=13, offset=1)
    plan = BlockPlan.from_mask(torch.from_numpy(mask).to(DEV), M, K, 128)
    want = 2 * (a.double() * _keep(mask, M, K)) @ b.double().T
    for shape in ((M, N), (N, (M + 3) // 4 * 4)):
        buf = torch.full(shape, float("nan"), device=DEV)
        out = buf if shape[0] == M else buf[:, :M].T
        dsd(a, b, plan, _lib.SD_PLAN_ROWS, 2.0, out=out)
        _check(out, want, torch.float16, f"fp32 {shape}")
    _check(GEMM().gemm(a, b), a.double() @ b.double().T, torch.float16, "dense")


def test_repeats_bit_for_bit(built_lib):
    from flash_dropout import _lib
    from flash_dropout.cuda.binding_gemm import BlockPlan, dsd
    a, b = _operands(2432, 1288, 1096, torch.bfloat16, 5)
    plan = BlockPlan.from_mask(torch.from_numpy(pm.block_mask(2432, 1096, 128, 0.3, seed=1, offset=2)).to(DEV), 2432, 1096, 128)
    first = dsd(a, b, plan, _lib.SD_PLAN_ROWS, 1.0)
    for _ in range(20):
        assert torch.equal(first, dsd(a, b, plan, _lib.SD_PLAN_ROWS, 1.0))

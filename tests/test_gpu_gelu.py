"""The GELU of the transformer consumers: every 16-bit input against fp64, ragged lengths, and what is left to torch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_input_against_fp64(built_lib, dtype):
    """Half an ulp of the result, plus 1e-6: the tail's approximation is good to 1.5e-7, its fp32 arithmetic adds a few ulps."""
    from flash_dropout.layers.gelu import GELU
    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype).to(DEV)
    x = x[torch.isfinite(x)].requires_grad_()
    dy = torch.randn(x.numel(), generator=torch.Generator().manual_seed(0)).to(dtype).to(DEV)
    y = GELU()(x)
    y.backward(dy)
    assert type(y.grad_fn).__name__ == "SparseDropGeluBackward" or y.grad_fn.name() == "SparseDropGeluBackward"
    ref = x.detach().double().requires_grad_()
    want = F.gelu(ref)
    want.backward(dy.double())
    ulp = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    for got, exact, scale in ((y.detach(), want.detach(), 1.0), (x.grad, ref.grad, dy.double().abs())):
        inside = exact.abs() < torch.finfo(dtype).max
        assert bool(((got.double() - exact).abs() <= ulp * exact.abs() + 1e-6 * scale + 1e-7)[inside].all())


@pytest.mark.parametrize("n", [1, 7, 8, 2047, 2048, 2049, 3 * 2048 + 13])
def test_ragged_lengths_and_special_values(built_lib, n):
    from flash_dropout.layers.gelu import GELU
    x = torch.randn(n, device=DEV).bfloat16()
    x[::5] = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0, -300.0], device=DEV).bfloat16().repeat(n)[: x[::5].numel()]
    got, want = GELU()(x), F.gelu(x)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    torch.testing.assert_close(got, want, rtol=2 ** -7, atol=1e-6, equal_nan=True)


def test_anything_else_is_torch(built_lib):
    from flash_dropout.layers.gelu import GELU
    gelu = GELU()
    x = torch.randn(64, 48, device=DEV)
    assert torch.equal(gelu(x), F.gelu(x))
    h = x.half()
    for t in (h.T, h.flatten()[1:], h[:0]):
        assert torch.equal(gelu(t), F.gelu(t))
    assert torch.equal(GELU(approximate="tanh")(h), F.gelu(h, approximate="tanh"))
    assert torch.equal(torch.func.vmap(gelu)(h), F.gelu(h))
    assert torch.equal(gelu(x.cpu()), F.gelu(x.cpu()))
    # the gradient's own graph
    a = h.clone().requires_grad_()
    (g,) = torch.autograd.grad(gelu(a).sum(), a, create_graph=True)
    g.sum().backward()
    assert a.grad is not None


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_no_result_is_further_off_than_torch(built_lib, dtype):
    """Over all finite 16-bit inputs, value and derivative against fp64: never further than torch's own kernels."""
    from flash_dropout.layers.gelu import GELU
    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype).to(DEV)
    x = x[torch.isfinite(x)]
    dy = torch.randn(x.numel(), generator=torch.Generator().manual_seed(1)).to(dtype).to(DEV)
    exact = x.double().requires_grad_()
    F.gelu(exact).backward(dy.double())
    sides = []
    for module in (GELU(), torch.nn.GELU()):
        a = x.clone().requires_grad_()
        y = module(a)
        y.backward(dy)
        sides.append((y.detach(), a.grad))
    for ours, torchs, want in zip(*sides, (F.gelu(x.double()), exact.grad)):
        inside = want.abs() < torch.finfo(dtype).max / 2
        further = (ours.double() - want).abs() > (torchs.double() - want).abs()
        assert not bool(further[inside].any()), f"{int(further[inside].sum())} of {x.numel()}"


def test_batched_and_dual_gradients_are_torch(built_lib):
    """A gradient that carries a batch dimension or a tangent of its own is differentiated by torch's operators."""
    import torch.autograd.forward_ad as fwad
    from flash_dropout.layers.gelu import GELU
    x = torch.randn(64, 48, device=DEV).half().requires_grad_()
    y = GELU()(x)
    dys = torch.randn(3, 64, 48, device=DEV).half()
    (got,) = torch.autograd.grad(y, x, dys, is_grads_batched=True, retain_graph=True)
    for g, dy in zip(got, dys):
        torch.testing.assert_close(g, torch.ops.aten.gelu_backward(dy, x.detach()))
    with fwad.dual_level():
        (g,) = torch.autograd.grad(y, x, fwad.make_dual(dys[0], dys[1]))
        value, tangent = fwad.unpack_dual(g)
    torch.testing.assert_close(value, torch.ops.aten.gelu_backward(dys[0], x.detach()))
    assert tangent is not None
    torch.testing.assert_close(tangent, torch.ops.aten.gelu_backward(dys[1], x.detach()))

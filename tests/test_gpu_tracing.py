"""What torch.jit.trace records of the native operators: the operation, not its result on the example."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _trace(fn, *example):
    return torch.jit.trace(fn, example, check_trace=False)


@pytest.mark.parametrize("grad", [False, True])
def test_layer_norm(built_lib, grad):
    from flash_dropout.layers.norm import LayerNorm
    norm = LayerNorm(256).to(DEV)
    with torch.set_grad_enabled(grad):
        traced = _trace(norm, torch.randn(8, 256, device=DEV))
        x = torch.randn(8, 256, device=DEV)
        torch.testing.assert_close(traced(x), TF.layer_norm(x, (256,), norm.weight, norm.bias, norm.eps))


def test_evaluated_gpt(built_lib):
    """Every layer of the evaluated model follows the new tokens (its own forward, 1e-4: fp32 LayerNorm kernels on one side)."""
    from flash_dropout.train import GPT
    torch.manual_seed(0)
    model = GPT(65, 32, 2, 2, 128, dict(p=0.2, variant="blockwise[cuda]", block_size=128)).to(DEV).eval()
    a, b = (torch.randint(0, 65, (2, 32), device=DEV) for _ in range(2))

    class Logits(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.model = model

        def forward(self, idx):
            return self.model(idx)[0]

    with torch.no_grad():
        traced = _trace(Logits().eval(), a)
        torch.testing.assert_close(traced(b), model(b)[0], rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("autocast", [False, True])
def test_linear(built_lib, autocast):
    """p = 0: the product of the new operands, and their gradients; with fp16 rounding on both sides (2e-3 of O(1) values)."""
    import flash_dropout.functional as F
    dt = torch.float32 if autocast else torch.float16
    make = lambda r: (torch.randn(r, 192, device=DEV) * 192 ** -0.25).to(dt)  # noqa: E731
    fn = lambda x, w: F.cuda_blockwise_dropout_matmul(x, w, 128, 0.0)  # noqa: E731
    with torch.autocast("cuda", dtype=torch.float16, enabled=autocast):
        traced = _trace(fn, make(256).requires_grad_(), make(136).requires_grad_())
        x, w = make(256).requires_grad_(), make(136).requires_grad_()
        y = traced(x, w)
    dy = torch.randn(256, 136, device=DEV).half() * 0.1
    y.backward(dy)
    tol = dict(rtol=2e-3, atol=2e-3)
    torch.testing.assert_close(y.float(), x.detach().half().float() @ w.detach().half().float().T, **tol)
    torch.testing.assert_close(x.grad.float(), dy.float() @ w.detach().half().float(), **tol)
    torch.testing.assert_close(w.grad.float(), dy.float().T @ x.detach().half().float(), **tol)


def test_a_traced_layer_draws_fresh_masks(built_lib):
    from flash_dropout import random as sd_random
    from flash_dropout.layers import DropoutMM
    layer = DropoutMM(1024, 128, p=0.5, variant="blockwise[cuda]", block_size=128).to(DEV).half()
    x = torch.ones(1024, 1024, device=DEV, dtype=torch.float16)
    sd_random.manual_seed(1, subsequence=0)
    try:
        traced = _trace(layer, x)
        a, b = traced(x), traced(x)
        assert not torch.equal(a, b)
    finally:
        sd_random.follow_torch_seed()


def test_conv(built_lib):
    import flash_dropout.functional as F
    make = lambda: (torch.randn(2, 16, 16, 16, device=DEV).half().requires_grad_(),  # noqa: E731
                    (torch.randn(24, 16, 3, 3, device=DEV) / 12).half().requires_grad_())
    fn = lambda x, k: F.cuda_blockwise_dropout_conv2d(x, k, 128, 0.0, padding=(1, 1))  # noqa: E731
    traced = _trace(fn, *make())
    x, k = make()
    y = traced(x, k)
    dy = torch.randn(y.shape, device=DEV).half() * 0.1
    y.backward(dy)
    xr, kr = x.detach().float().requires_grad_(), k.detach().float().requires_grad_()
    want = TF.conv2d(xr, kr, padding=1)
    want.backward(dy.float())
    tol = dict(rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(y.float(), want, **tol)
    torch.testing.assert_close(x.grad.float(), xr.grad, **tol)
    torch.testing.assert_close(k.grad.float(), kr.grad, **tol)

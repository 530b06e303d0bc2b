"""The residual sum: bit for bit torch's, with its gradients, at ragged lengths, and what is left to torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1,), (7,), (8,), (3, 683), (1, 2048), (2, 5, 411)])
def test_against_torch(built_lib, dtype, shape):
    from flash_dropout.layers.residual import residual_add
    x = torch.randn(shape, device=DEV, requires_grad=True)
    r = torch.randn(shape, device=DEV).to(dtype).requires_grad_()
    dy = torch.randn(shape, device=DEV)
    y = residual_add(x, r)
    assert y.grad_fn.name() == "SparseDropResidualBackward"
    got = (y, *torch.autograd.grad(y, (x, r), dy))
    want = x + r
    for a, b in zip(got, (want, *torch.autograd.grad(want, (x, r), dy))):
        assert a.dtype == b.dtype and torch.equal(a, b)


def test_anything_else_is_torch(built_lib):
    from flash_dropout.layers.residual import residual_add
    x, h = torch.randn(16, 24, device=DEV), torch.randn(16, 24, device=DEV).half()
    for a, b in ((x, x), (h, h), (h, x), (x, h[0]), (x.T, h.T), (x[:, 1:], h[:, 1:]), (x.cpu(), h.cpu()), (x[:0], h[:0])):
        y = residual_add(a, b)
        assert torch.equal(y, a + b) and y.dtype == (a + b).dtype
    assert torch.equal(torch.func.vmap(residual_add)(x, h), x + h)
    with pytest.raises(RuntimeError):
        residual_add(x, h.cpu())

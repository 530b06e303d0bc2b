"""What backward makes of saved tensors that hooks have packed: any strides, but no other type, device or shape."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _linear(x):
    import flash_dropout.functional as F
    w = (torch.randn(136, 128, generator=torch.Generator(DEV).manual_seed(2), device=DEV) * 0.1).half().requires_grad_()
    return F.cuda_blockwise_dropout_matmul(x, w, 128, 0.5, relu=True, any_rank=True), (x, w)


def _conv(x, **more):
    import flash_dropout.functional as F
    k = (torch.randn(24, x.size(1), 3, 3, generator=torch.Generator(DEV).manual_seed(2), device=DEV) * 0.1).half().requires_grad_()
    return F.cuda_blockwise_dropout_conv2d(x, k, 128, 0.5, padding=(1, 1), **more), (x, k)


def _norm(x):
    from flash_dropout.layers.norm import LayerNorm
    norm = LayerNorm(x.size(-1)).to(DEV)
    return norm(x), (x, norm.weight, norm.bias)


def _gelu(x):
    from flash_dropout.layers.gelu import GELU
    return GELU()(x), (x,)


CASES = {
    "linear": (_linear, (2, 96, 128), torch.float16),
    "linear 2-D": (_linear, (192, 128), torch.float16),
    "conv": (_conv, (2, 16, 16, 16), torch.float16),
    "conv unfused": (lambda x: _conv(x, fused=False), (2, 16, 16, 16), torch.float16),
    "norm": (_norm, (3, 64, 96), torch.float32),
    "gelu": (_gelu, (3, 64, 96), torch.bfloat16),
}


def _gradients(name, pack, unpack):
    from flash_dropout import random as sd_random
    fn, shape, dt = CASES[name]
    g = torch.Generator(DEV).manual_seed(1)
    x = torch.randn(shape, generator=g, device=DEV).to(dt).requires_grad_()
    sd_random.manual_seed(4, subsequence=0)
    try:
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            y, leaves = fn(x)
    finally:
        sd_random.follow_torch_seed()
    y.backward(torch.randn(y.shape, generator=g, device=DEV).to(y.dtype))
    return [t.grad for t in leaves]


def _keep(t):
    return t


def _other_strides(t):
    if t.dim() < 2:
        return t
    return t.transpose(-1, -2).contiguous().transpose(-1, -2)


def _off_boundary(t):
    return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("unpack", [_other_strides, _off_boundary])
def test_strides_and_alignment(built_lib, name, unpack):
    """Bit for bit; the LayerNorm's parameter gradients add the partial sums of a CTA's eight warps in the order in which they
    arrive, so those agree to 8 * 2^-24 of the sum of their 192 terms' magnitudes (about 150)."""
    atol = 8 * 2 ** -24 * 200 if name == "norm" else 0
    for a, b in zip(_gradients(name, _keep, _keep), _gradients(name, _keep, unpack)):
        torch.testing.assert_close(a, b, rtol=0, atol=atol)


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("unpack", [lambda t: t.cpu(), lambda t: t.double(), lambda t: t.flatten()[1:], lambda t: t.unsqueeze(0)],
                         ids=["device", "type", "elements", "shape"])
def test_anything_else_is_refused(built_lib, name, unpack):
    with pytest.raises(RuntimeError, match="came back from its hooks"):
        _gradients(name, _keep, unpack)

"""CUDA graphs that share tensors with one another and with eager calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _product(x, w):
    """p = 0 under fp16 autocast: x . w^T, from operands in fp32."""
    import flash_dropout.functional as F
    with torch.autocast("cuda", dtype=torch.float16):
        return F.cuda_blockwise_dropout_matmul(x, w, 128, 0.0)


def _close(y, x, w):
    torch.testing.assert_close(y.float(), x.half().float() @ w.detach().half().float().T, rtol=2e-3, atol=2e-3)


@pytest.fixture
def operands():
    x = torch.randn(256, 128, device=DEV) * 128 ** -0.25
    ws = [(torch.randn(128, 128, device=DEV) * 128 ** -0.25).requires_grad_() for _ in range(2)]
    for w in ws:
        _product(x, w)                                  # everything that is made once exists
    torch.cuda.synchronize()
    return x, ws


def test_a_graph_casts_its_own_inputs(built_lib, operands):
    """Two graphs over one static fp32 input, the first one's result kept: the second replays alone, on new values."""
    x, (wa, wb) = operands
    g1, g2 = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g1):
        y1 = _product(x, wa)                            # its node keeps the 16-bit copy of x
    with torch.cuda.graph(g2):
        y2 = _product(x, wb)
    x.copy_(torch.randn_like(x) * 128 ** -0.25)
    g2.replay()
    _close(y2, x, wb)
    g1.replay()
    _close(y1, x, wa)


def test_an_eager_call_after_a_capture(built_lib, operands):
    x, (wa, wb) = operands
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        y1 = _product(x, wa)
    with torch.cuda.stream(s):
        y2 = _product(x, wb)                            # the capture has run nothing yet
    torch.cuda.current_stream().wait_stream(s)
    _close(y2, x, wb)
    g.replay()
    _close(y1, x, wa)


def test_a_tensor_that_a_replay_writes(built_lib, operands):
    """A replay leaves no trace on the tensors it writes; eager layers behind it see the new values."""
    x, (wa, wb) = operands
    src = x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        h = src * 2
    g.replay()
    y1 = _product(h, wa)
    _close(y1, h, wa)
    src.copy_(torch.randn_like(src) * 128 ** -0.25)
    g.replay()
    y2 = _product(h, wb)
    _close(y2, h, wb)

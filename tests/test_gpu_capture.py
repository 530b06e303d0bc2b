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


def _long(seed):
    """Operands of a product that is cut along its reduction: two tiles, 32 K tiles."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    return tuple((torch.randn(256, 4096, generator=g, device=DEV) * 4096 ** -0.25).half() for _ in range(2))


def test_every_graph_has_a_workspace_of_its_own(built_lib):
    """Cleared by its own replay, not by that of an earlier graph: the second one replays first."""
    import flash_dropout
    import flash_dropout.functional as F
    from flash_dropout.cuda import binding_gemm as bg
    graphs = []
    for i in range(2):
        x, w = _long(i)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = F.cuda_blockwise_dropout_matmul(x, w, 128, 0.0)
            where = bg.workspace(DEV).data_ptr()
            assert where == bg.workspace(DEV).data_ptr()
        graphs.append((g, x, w, y, where))
    assert graphs[0][4] != graphs[1][4]
    for g, x, w, y, _ in (graphs[1], graphs[0], graphs[1]):
        y.zero_()
        g.replay()
        torch.testing.assert_close(y.float(), x.float() @ w.float().T, rtol=2e-3, atol=2e-2)
    flash_dropout.check_status(DEV)


def test_the_status_word_of_a_first_launch_in_a_capture():
    """In a process whose first launch is captured the word is zero before the first replay, and no replay clears it."""
    import os
    import subprocess
    import sys
    code = """
import torch, flash_dropout.functional as F
from flash_dropout.cuda import binding_gemm as bg
dev = torch.device("cuda:0")
x = torch.ones(128, 128, device=dev, dtype=torch.float16)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    y = F.cuda_blockwise_dropout_matmul(x, x, 128, 0.0)
word = bg.status_word(dev)
assert word.tolist() == [0, 0, 0, 0], word.tolist()
word[3] = 7
g.replay()
assert word.tolist() == [0, 0, 0, 7], word.tolist()
assert bool((y == 128).all())
"""
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparse-dropout_b200")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=dict(os.environ, PYTHONPATH=path))


def test_weights_between_a_capture_and_its_first_replay(built_lib):
    """A step that updates outside its graph: until the first replay the 16-bit copies that the graph makes are those of the
    warm-up's last step, so an eager forward casts the weights itself."""
    from flash_dropout import random as sd_random
    from flash_dropout.train import BasicNet, FlatGradDataParallel, GraphedTrainStep
    torch.manual_seed(0)
    model = BasicNet(256, 1, 256, 10, dict(p=0.5, variant="blockwise[cuda]", block_size=128)).to(DEV)
    x, y = torch.rand(256, 256, device=DEV), torch.randint(0, 10, (256,), device=DEV)
    dp = FlatGradDataParallel(model, fuse_wgrad=True)
    dp.shadow_min_layers = 1
    opt = torch.optim.AdamW(model.parameters(), lr=1e-1)
    sd_random.manual_seed(3, subsequence=0)
    try:
        GraphedTrainStep(model, dp, opt, lambda m, a, b: torch.nn.functional.cross_entropy(m(a).float(), b), (x, y),
                         autocast_dtype=torch.bfloat16, whole_step=False)
        outs = []
        for copies in (True, False):
            for p in dp._shadow_params:
                p._sd_w16 = p._sd_w16 if copies else None
            sd_random.device_counter(DEV).zero_()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                outs.append(model(x).detach())
        assert torch.equal(*outs)
    finally:
        sd_random.disable_device_counter()
        sd_random.follow_torch_seed()

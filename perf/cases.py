"""The workloads on which this framework's speed is measured: what its users run, through the public entry points.

A case is a dict of plain values; ``kind`` says which entry point it goes through:

  linear   one SparseDrop linear, forward and backward: ``flash_dropout.functional.cuda_blockwise_dropout_matmul`` on
           16-bit tensors, or with ``layer`` a ``flash_dropout.layers.DropoutMM`` under autocast on fp32 activations.
           ``backward`` False is the forward alone, as in Monte-Carlo dropout at inference.
  gemm     the extension-style wrapper ``GEMM`` with an explicit block mask: the three products of a linear layer
  conv     ``cuda_blockwise_dropout_conv2d`` (``layer``: ``DropoutConv2d`` under autocast), forward and backward
  mlp/gpt  one training step (zero grad, forward, backward, AdamW) of ``BasicNet`` or ``GPT``: captured in a CUDA graph
           (``graph`` True: ``GraphedTrainStep``) or launched eagerly (``train_step``)

Every pass draws its block masks itself (except ``gemm``, which is given one), from a stream that ``prepare`` seeds.
"""
import math
import os
import sys

import torch

# the package of the tree that runs this file: the working folder
sys.path.insert(0, os.path.join(os.getcwd(), "sparse-dropout_b200"))

import flash_dropout.functional as F  # noqa: E402
from flash_dropout import random as sd_random  # noqa: E402
from flash_dropout.cuda.binding_gemm import GEMM  # noqa: E402
from flash_dropout.layers import DropoutConv2d, DropoutMM  # noqa: E402
from flash_dropout.train import GPT, BasicNet, FlatGradDataParallel, GraphedTrainStep, train_step  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _linear(M, N, K, p, dtype, **more):
    return dict(dict(kind="linear", M=M, N=N, K=K, p=p, dtype=dtype, block=128, layer=False, backward=True), **more)


def _gemm(M, N, K, p, dtype):
    return dict(kind="gemm", M=M, N=N, K=K, p=p, dtype=dtype, block=128)


def _conv(N, C, H, W, Ko, R, S, stride, pad, dilation, p, dtype, layer=False):
    return dict(kind="conv", N=N, C=C, H=H, W=W, Ko=Ko, R=R, S=S, stride=stride, pad=pad, dilation=dilation, p=p,
                dtype=dtype, layer=layer)


def _mlp(batch, inputs, hidden, layers, p, dtype, graph):
    return dict(kind="mlp", batch=batch, inputs=inputs, hidden=hidden, layers=layers, p=p, dtype=dtype, graph=graph)


def _gpt(batch, ctx, n_layer, n_head, n_embed, p, dtype, graph):
    return dict(kind="gpt", batch=batch, ctx=ctx, n_layer=n_layer, n_head=n_head, n_embed=n_embed, p=p, dtype=dtype,
                graph=graph)


def listed():
    return [
        # the small end of the operator's test grid: a small layer called eagerly, where launches and host time count
        dict(_linear(512, 512, 512, 0.5, "fp16"), name="linear 512"),
        # the size at which the method's report compares layers (forward + backward, 1024 cubed)
        dict(_linear(1024, 1024, 1024, 0.5, "fp16"), name="linear 1024"),
        # an odd batch through odd widths: nothing is a multiple of the 128-wide block
        dict(_linear(2500, 1352, 3016, 0.3, "bf16"), name="linear ragged"),
        # the headline layer of the benchmark
        dict(_linear(4096, 4096, 4096, 0.5, "fp16"), name="linear 4096"),
        # a wide layer fed a large token batch, light dropout: the largest products
        dict(_linear(16384, 4096, 4096, 0.2, "bf16"), name="linear 16384x4096"),
        # the first MLP linear of the char-GPT as a module under autocast, 64 x 256 tokens
        dict(_linear(16384, 1536, 384, 0.2, "bf16", layer=True), name="layer gpt c_fc"),
        # code written against the reference's extension: explicit mask, three products
        dict(_gemm(2048, 2048, 2048, 0.5, "fp16"), name="gemm wrapper 2048"),
        # the benchmark's convolution: 3x3, 64 -> 128 channels, 32x32 images, batch 256
        dict(_conv(256, 64, 32, 32, 128, 3, 3, 1, 1, 1, 0.5, "fp16"), name="conv 3x3"),
        # a down-sampling convolution of an image network on 56x56 maps, as a module under autocast
        dict(_conv(64, 64, 56, 56, 128, 3, 3, 2, 1, 1, 0.3, "bf16", layer=True), name="conv strided"),
        # the MLP training step at the benchmark's size, captured once and replayed
        dict(_mlp(512, 784, 1024, 2, 0.5, "bf16", True), name="mlp step graph"),
        # the same model stepped eagerly, as in a plain training loop
        dict(_mlp(512, 784, 1024, 2, 0.5, "bf16", False), name="mlp step eager"),
        # the char-GPT training step at the benchmark's size, captured once and replayed
        dict(_gpt(64, 256, 6, 6, 384, 0.2, "bf16", True), name="gpt step graph"),
    ]


def _log(rng, lo, hi, step=1):
    """An integer between lo and hi, spread over its logarithm, a multiple of ``step``."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "gemm", "conv", "conv", "mlp", "gpt"])
    p = rng.choice([0.0, 0.1, 0.2, 0.3, 0.5, 0.5, 0.7, 0.9])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("linear", "gemm"):
        while True:      # rows any number, widths multiples of 8 (the operator's rule), half of them round
            if rng.random() < 0.5:
                M, N, K = _log(rng, 128, 16384, 128), _log(rng, 128, 8192, 128), _log(rng, 128, 8192, 128)
            else:
                M, N, K = _log(rng, 100, 16384), _log(rng, 104, 8192, 8), _log(rng, 104, 8192, 8)
            if kind == "gemm":
                M = (M + 7) // 8 * 8             # x^T as an operand: 16-byte rows
            if M * N * K * (1 - p) <= 16384 * 4096 * 4096 * 0.8:
                break
        if kind == "gemm":
            return _gemm(M, N, K, p, dtype)
        return _linear(M, N, K, p, dtype, block=rng.choice([128, 128, 128, 256]), layer=rng.random() < 0.4,
                       backward=rng.random() < 0.8)
    if kind == "conv":
        while True:
            R = rng.choice([1, 3, 3, 3, 3, 5])
            H, C, Ko = rng.choice([7, 8, 14, 16, 28, 32, 32, 56, 64]), _log(rng, 16, 256, 8), _log(rng, 16, 256, 8)
            stride, N = rng.choice([1, 1, 1, 2]), _log(rng, 16, 256)
            if N * H * H * C * Ko * R * R <= 4 * 256 * 32 * 32 * 64 * 128 * 9 and N * H * H * max(C, Ko) <= 1 << 26:
                break
        return _conv(N, C, H, H, Ko, R, R, stride, R // 2, 1, p, dtype, layer=rng.random() < 0.4)
    if kind == "mlp":
        return _mlp(_log(rng, 64, 4096, 8), _log(rng, 256, 3072, 8), _log(rng, 256, 2048, 128), rng.randint(1, 4), p, dtype,
                    rng.random() < 0.5)
    heads = rng.choice([4, 6, 8, 12])
    return _gpt(_log(rng, 4, 64), rng.choice([64, 128, 256]), rng.randint(2, 6), heads, 64 * heads, p, dtype,
                rng.random() < 0.5)


def _weight(shape, fan_in, g, dtype, dev):
    """The layers' own initialisation: uniform within 1 / sqrt(fan_in)."""
    return ((torch.rand(shape, generator=g, device=dev) * 2 - 1) / math.sqrt(fan_in)).to(dtype)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    kind = case["kind"]
    torch.manual_seed(seed)
    sd_random.disable_device_counter(dev)
    sd_random.manual_seed(seed, subsequence=0)
    s = dict(case=dict(case), dt=dt)
    if kind in ("linear", "gemm"):
        M, N, K = case["M"], case["N"], case["K"]
        x = torch.randn(M, K, generator=g, device=dev)
        if kind == "linear" and case["layer"]:
            s["layer"] = DropoutMM(K, N, p=case["p"], variant="blockwise[cuda]", block_size=(case["block"],) * 2).to(dev)
            s["x"] = x.requires_grad_(case["backward"])
        else:
            grad = kind == "linear" and case["backward"]
            s["x"] = x.to(dt).requires_grad_(grad)
            s["w"] = _weight((N, K), K, g, dt, dev).requires_grad_(grad)
        s["dy"] = torch.randn(M, N, generator=g, device=dev).to(dt)
        if kind == "gemm":
            b = case["block"]
            s["mask"] = torch.rand(-(-M // b), -(-K // b), generator=g, device=dev) < case["p"]
    elif kind == "conv":
        N, C, H, W, Ko, R, S = (case[k] for k in ("N", "C", "H", "W", "Ko", "R", "S"))
        P, Q = _conv_out(case)
        x = torch.randn(N, C, H, W, generator=g, device=dev)
        geom = dict(padding=(case["pad"],) * 2, stride=(case["stride"],) * 2, dilation=(case["dilation"],) * 2)
        if case["layer"]:
            s["layer"] = DropoutConv2d(C, Ko, (R, S), p=case["p"], variant="blockwise[cuda]", block_size=128, **geom).to(dev)
            s["x"] = x.requires_grad_()
        else:
            s["x"] = x.to(dt).requires_grad_()
            s["w"] = _weight((Ko, C, R, S), C * R * S, g, dt, dev).requires_grad_()
            s["geom"] = geom
        # gradients of the layers that follow come in the memory format of the convolution's own result
        s["dy"] = torch.randn(N, P, Q, Ko, generator=g, device=dev).to(dt).permute(0, 3, 1, 2)
    else:
        dropout = dict(p=case["p"], variant="blockwise[cuda]", block_size=(128, 128))
        if kind == "mlp":
            model = BasicNet(case["inputs"], case["layers"], case["hidden"], 10, dropout).to(dev)
            opt = torch.optim.AdamW(model.parameters(), lr=1e-3, fused=True)
            s["inputs"] = (torch.rand(case["batch"], case["inputs"], generator=g, device=dev),
                           torch.randint(0, 10, (case["batch"],), generator=g, device=dev))
            s["loss_of"] = lambda m, a, b: torch.nn.functional.cross_entropy(m(a).float(), b)
        else:
            model = GPT(65, case["ctx"], case["n_layer"], case["n_head"], case["n_embed"], dropout).to(dev)
            opt = model.configure_optimizers(weight_decay=0.1, lr=3e-4)
            s["inputs"] = (torch.randint(0, 65, (case["batch"], case["ctx"]), generator=g, device=dev),)
            s["loss_of"] = lambda m, a: m(a)[1]
        dp = FlatGradDataParallel(model, fuse_wgrad=True)
        sd_random.manual_seed(seed, subsequence=0)
        s.update(model=model, opt=opt, dp=dp)
        if case["graph"]:
            s["counter"] = sd_random.enable_device_counter(dev)      # the captured step keeps drawing from this counter
            start = [q.detach().clone() for q in model.parameters()]
            s["step"] = GraphedTrainStep(model, dp, opt, s["loss_of"], s["inputs"], autocast_dtype=dt)
            with torch.no_grad():                # the capture's warm-up has trained: back to the start, in place
                torch._foreach_copy_(list(model.parameters()), start)
                for moments in opt.state.values():
                    for t in moments.values():
                        t.zero_()
                s["counter"].zero_()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gemm":
        lib, x, w, dy, mask, b = GEMM(), state["x"], state["w"], state["dy"], state["mask"], case["block"]
        scale = 1 / (1 - case["p"])
        y = lib.gemm_dsd(x, w, mask, b, scale)
        dx = lib.gemm_sdd(dy, w.T, mask, b, scale)
        dw = lib.gemm_dsd(x.T, dy.T, mask.T, b, scale)
        return dict(y=y, dx=dx, dw=dw)
    if kind == "linear" and not case["backward"]:
        with torch.no_grad():
            if case["layer"]:
                with torch.autocast("cuda", dtype=state["dt"]):
                    return dict(y=state["layer"](state["x"]))
            return dict(y=F.cuda_blockwise_dropout_matmul(state["x"], state["w"], case["block"], case["p"]))
    if kind in ("linear", "conv"):
        x = state["x"]
        if case["layer"]:
            w = state["layer"].weight
            with torch.autocast("cuda", dtype=state["dt"]):
                y = state["layer"](x)
        elif kind == "linear":
            w = state["w"]
            y = F.cuda_blockwise_dropout_matmul(x, w, case["block"], case["p"])
        else:
            w = state["w"]
            y = F.cuda_blockwise_dropout_conv2d(x, w, 128, case["p"], **state["geom"])
        x.grad = w.grad = None
        y.backward(state["dy"])
        return dict(y=y.detach(), dx=x.grad, dw=w.grad)
    if case["graph"]:
        loss = state["step"]()
    else:
        loss_of, inputs = state["loss_of"], state["inputs"]
        loss = train_step(state["model"], state["dp"], state["opt"], lambda m: loss_of(m, *inputs), autocast_dtype=state["dt"])
    return dict(loss=loss, grad=state["dp"].flat_grad, params=[q.detach() for q in state["model"].parameters()])


def _conv_out(case):
    out = lambda n, k: (n + 2 * case["pad"] - case["dilation"] * (k - 1) - 1) // case["stride"] + 1  # noqa: E731
    return out(case["H"], case["R"]), out(case["W"], case["S"])


def work(case):
    """Floating-point operations on kept blocks, and every input read and output written once."""
    kind, keep = case["kind"], 1 - case["p"]
    if kind in ("linear", "gemm"):
        M, N, K = case["M"], case["N"], case["K"]
        wide = 4 if case.get("layer") else 2               # bytes of activations and weights where they are kept in fp32
        if not case.get("backward", True):
            return {"bytes": wide * (M * K * keep + N * K) + 2 * M * N, "flops": 2.0 * M * N * K * keep}
        return {"bytes": wide * (M * K * (keep + 1) + 2 * N * K) + 2 * 2 * M * N, "flops": 6.0 * M * N * K * keep}
    if kind == "conv":
        P, Q = _conv_out(case)
        rows, cols = case["N"] * P * Q, case["C"] * case["R"] * case["S"]
        wide = 4 if case["layer"] else 2
        return {"bytes": wide * 2 * (case["N"] * case["C"] * case["H"] * case["W"] + case["Ko"] * cols) + 2 * 2 * rows * case["Ko"],
                "flops": 6.0 * rows * cols * case["Ko"] * keep}
    # training steps: parameters and both moments read and written, gradients written, the batch read
    if kind == "mlp":
        B, I, Hd, L = case["batch"], case["inputs"], case["hidden"], case["layers"]
        params = I * Hd + L * Hd * Hd + Hd * 128
        return {"bytes": 28 * params + 4 * B * I, "flops": B * keep * (4.0 * I * Hd + 6.0 * (L * Hd * Hd + Hd * 128))}
    T, d, L = case["batch"] * case["ctx"], case["n_embed"], case["n_layer"]
    params = 12 * L * d * d + (2 * 65 + case["ctx"]) * d
    attention = 7.0 * case["ctx"] * d * L * T              # causal scores and values, forward and backward
    return {"bytes": 28 * params + 8 * T, "flops": 6.0 * T * (12 * L * d * d * keep + 65 * d) + attention}


def tolerance(case):
    # one rounding to the 16-bit result of sums taken in fp32; training steps: the same rounding carried through the
    # layers, and through the first AdamW updates, which take the sign of gradients that are all rounding (the masked-
    # dense layers in plain PyTorch on the same masks: gradient of the second step within 0.012 of the kernels' one)
    if case["kind"] in ("mlp", "gpt"):
        return {"rel": 0.02, "max": 0.9}
    return {"rel": 2e-3, "max": 1e-2} if case["dtype"] == "fp16" else {"rel": 1e-2, "max": 5e-2}

"""The one-launch AdamW of the training steps against torch's own optimizer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("sizes", [[1], [2047, 2048, 2049], [5, 3, 4096 * 3 + 1, 300_003]])
@pytest.mark.parametrize("capturable", [False, True])
def test_adamw_matches_torch(built_lib, sizes, capturable):
    """Five steps with two parameter groups and changing gradients and learning rate.  Both sides evaluate the same formula
    in fp32; the few roundings per step that may fall differently move a parameter by at most ~4 ulp of its update
    (4 * 2^-23 * lr per step), far below the bound, and the moments by ulps."""
    from flash_dropout.train.dp import _FusedAdamW
    g = torch.Generator().manual_seed(sum(sizes))
    start = [torch.randn(n, generator=g) for n in sizes]
    grads = [[torch.randn(n, generator=g) * 10.0 ** -k for n in sizes] for k in range(5)]
    sides = []
    for ours in (False, True):
        params = [torch.nn.Parameter(t.to(DEV)) for t in start]
        groups = [{"params": params[:1], "weight_decay": 0.1}, {"params": params[1:], "weight_decay": 0.0}]
        opt = torch.optim.AdamW([gr for gr in groups if gr["params"]], lr=1e-2, fused=True, capturable=capturable)
        # every gradient 16-byte aligned, as the kernel asks; a misaligned one takes torch's step
        for p in params:
            p.grad = torch.zeros_like(p)
        fused = _FusedAdamW()
        for k in range(5):
            for gr in opt.param_groups:
                gr["lr"] = 1e-2 / (k + 1)
            for p, t in zip(params, grads[k]):
                p.grad.copy_(t)
            fused.step(opt) if ours else opt.step()
        assert not ours or fused._native is not None
        sides.append([(p.detach(), *(opt.state[p][k] for k in ("exp_avg", "exp_avg_sq", "step"))) for p in params])
    for a, b in zip(*sides):
        assert torch.equal(a[3], b[3]) and a[3].item() == 5
        for x, y in zip(a[:3], b[:3]):
            torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-7)


def test_anything_else_is_left_to_the_optimizer(built_lib):
    from flash_dropout.train.dp import _FusedAdamW
    p = torch.nn.Parameter(torch.ones(8, device=DEV))
    p.grad = torch.ones_like(p)
    for make in (lambda: torch.optim.AdamW([p], amsgrad=True), lambda: torch.optim.Adam([p]), lambda: torch.optim.SGD([p], lr=0.1)):
        opt, fused = make(), _FusedAdamW()
        before = p.detach().clone()
        for _ in range(2):
            fused.step(opt)
        assert fused._native is None and not torch.equal(before, p)
    opt, fused = torch.optim.AdamW([p], lr=0.1, fused=True), _FusedAdamW()
    for _ in range(2):
        fused.step(opt)
    assert fused._native is not None
    opt.load_state_dict(opt.state_dict())                  # new state tensors: described again, not updated through stale pointers
    steps = opt.state[p]["step"]
    fused.step(opt)
    assert steps.item() == 3


def test_a_model_that_has_been_stepped_is_freed(built_lib):
    """The optimizer's description must not keep parameters alive: they lead back to it through their gradient hooks."""
    import gc
    import weakref
    from flash_dropout.train import BasicNet, FlatGradDataParallel, train_step
    model = BasicNet(128, 2, 128, 10, dict(p=0.5, variant="blockwise[cuda]", block_size=128)).to(DEV)
    dp = FlatGradDataParallel(model)
    opt = torch.optim.AdamW(model.parameters(), lr=1e-3, fused=True)
    x = torch.randn(128, 128, device=DEV)
    for _ in range(3):
        train_step(model, dp, opt, lambda m: m(x).square().mean(), autocast_dtype=torch.bfloat16)
    assert dp.adamw._native is not None
    gone = [weakref.ref(dp), weakref.ref(model)]
    del model, dp, opt
    gc.collect()
    assert all(r() is None for r in gone)


@pytest.mark.parametrize("groups", [[[], [8]], [[8], []], [[], []]])
def test_empty_groups(built_lib, groups):
    """What a decay / no-decay split can leave behind is stepped as by the optimizer alone."""
    from flash_dropout.train.dp import _FusedAdamW
    sides = []
    for ours in (False, True):
        params = [[torch.nn.Parameter(torch.ones(n, device=DEV)) for n in ns] for ns in groups]
        opt = torch.optim.AdamW([dict(params=ps) for ps in params], lr=0.1, fused=True)
        fused = _FusedAdamW()
        for k in range(3):
            for p in sum(params, []):
                p.grad = torch.full_like(p, k + 1.0) if p.grad is None else p.grad.fill_(k + 1.0)
            fused.step(opt) if ours else opt.step()
        sides.append(sum(params, []))
    for a, b in zip(*sides):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("sizes", [[0, 8], [8, 0]])
def test_parameters_without_elements(built_lib, sizes):
    """The kernel's table has no place for them: the optimizer steps such a model by itself."""
    from flash_dropout.train.dp import _FusedAdamW
    params = [torch.nn.Parameter(torch.ones(n, device=DEV)) for n in sizes]
    opt, fused = torch.optim.AdamW(params, lr=0.1, fused=True), _FusedAdamW()
    for p in params:
        p.grad = torch.ones_like(p)
    for _ in range(3):
        fused.step(opt)
    assert fused._native is None and all(opt.state[p]["step"].item() == 3 for p in params)


def _one_step(p, g, m, v, t, lr, decay, b1=0.9, b2=0.999, eps=1e-8):
    p = p * (1 - lr * decay)
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    return p - lr / (1 - b1 ** t) * m / (v.sqrt() / (1 - b2 ** t) ** 0.5 + eps), m, v


@pytest.mark.parametrize("lr,decay", [(1e-3, 0.01), (1e-2, 0.0)])
def test_an_update_is_as_precise_as_torchs(built_lib, lr, decay):
    """Largest and rms error of one step against fp64 from the same state, over half a million elements; 5 % for the statistics
    of rounding."""
    from flash_dropout.train.dp import _FusedAdamW
    errors = []
    for ours in (False, True):
        gen = torch.Generator(device=DEV).manual_seed(7)
        p = torch.nn.Parameter(torch.randn(1 << 19, generator=gen, device=DEV) * 0.03)
        p.grad = torch.zeros_like(p)
        opt, fused = torch.optim.AdamW([p], lr=lr, weight_decay=decay, fused=True, capturable=True), _FusedAdamW()
        for k in range(5):
            p.grad.copy_(torch.randn(p.shape, generator=gen, device=DEV) * 10.0 ** -k)
            st = opt.state[p]
            before = [t.detach().double() for t in (p, p.grad, *(st.get(n, torch.zeros_like(p)) for n in ("exp_avg", "exp_avg_sq")))]
            fused.step(opt) if ours else opt.step()
        want = _one_step(*before, 5, lr, decay)
        err = [(a.detach().double() - b).abs() for a, b in zip((p, st["exp_avg"], st["exp_avg_sq"]), want)]
        errors.append([(e.max().item(), e.square().mean().sqrt().item()) for e in err])
    for theirs, mine, name in zip(*errors, ("p", "exp_avg", "exp_avg_sq")):
        assert all(b <= 1.05 * a for a, b in zip(theirs, mine)), (name, theirs, mine)

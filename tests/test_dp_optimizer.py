"""When the training steps look at an optimizer's tensors for the one-launch update (no GPU: nothing is launched)."""
import torch


def _with_cuda(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)


def test_an_empty_first_group(monkeypatch):
    from flash_dropout.train.dp import _FusedAdamW
    p = torch.nn.Parameter(torch.ones(8))
    p.grad = torch.ones(8)
    opt = torch.optim.AdamW([dict(params=[], weight_decay=0.1), dict(params=[p], weight_decay=0.0)], lr=0.1)
    with monkeypatch.context() as m:
        _with_cuda(m)
        for _ in range(2):
            _FusedAdamW().step(opt)
    assert opt.state[p]["step"].item() == 2 and bool((p < 1).all())


def test_an_optimizer_that_cannot_be_described_is_looked_at_ever_less_often(monkeypatch):
    """The walk over its tensors is repeated after 1, 2, 4, ... 64 steps, and at once after it has been of use."""
    from flash_dropout.train.dp import _FusedAdamW
    p = torch.nn.Parameter(torch.ones(8))
    p.grad = torch.ones(8)
    opt, fused, looked = torch.optim.AdamW([p], lr=0.1), _FusedAdamW(), []
    monkeypatch.setattr(fused, "_describe", lambda optimizer: looked.append(int(opt.state[p]["step"].item() if opt.state else 0)) or False)
    with monkeypatch.context() as m:
        _with_cuda(m)
        for _ in range(260):
            fused.step(opt)
    assert looked == [0, 1, 3, 7, 15, 31, 63, 127, 191, 255] and opt.state[p]["step"].item() == 260

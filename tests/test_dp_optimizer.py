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

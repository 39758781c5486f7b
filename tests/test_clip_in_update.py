"""Clipping inside the optimizer's own pass: the same weights as scaling the gradients first, and only where nothing could
look at the gradients in between."""
import pytest
import torch

from cubework_b200.engine import Trainer
from cubework_b200.global_vars import env
from cubework_b200.optim import FusedAdamW, FusedSGD, linear_warmup_schedule
from cubework_b200.utils.clip_grad import clip_grad_norm


def _model():
    env.load(mode=None)
    torch.manual_seed(0)
    return torch.nn.Sequential(torch.nn.Linear(12, 20), torch.nn.Tanh(), torch.nn.Linear(20, 3))


def _trainer(model, opt, **kw):
    crit = lambda out, target: ((out - target)**2).sum()
    return Trainer(model, crit, opt, amp_dtype=None, forward_fn=lambda m, b: (m(b["x"]), b["y"]), **kw)


@pytest.mark.parametrize("make", [lambda p: FusedAdamW(p, lr=1e-2), lambda p: FusedSGD(p, lr=1e-2, momentum=0.9)])
@pytest.mark.parametrize("clip", [0.1, 1e6])
def test_same_weights_as_scaling_first(make, clip):
    a, b = _model(), _model()
    b.load_state_dict(a.state_dict())
    oa, ob = make(a.parameters()), make(b.parameters())
    tr = _trainer(a, oa, clip=clip, lr_scheduler=linear_warmup_schedule(oa, 2, 10))
    sched = linear_warmup_schedule(ob, 2, 10)
    for i in range(4):
        g = torch.Generator().manual_seed(i)
        batch = dict(x=torch.randn(8, 12, generator=g), y=torch.randn(8, 3, generator=g))
        assert tr._folds_clipping()
        tr.step(batch)
        ((b(batch["x"]) - batch["y"])**2).sum().backward()
        clip_grad_norm(list(b.parameters()), clip)
        ob.step()
        sched.step()
        ob.zero_grad(set_to_none=True)
        for p, q in zip(a.parameters(), b.parameters()):
            assert torch.equal(p, q)             # both multiply the fp32 gradient by the factor once


def test_not_where_the_gradients_can_be_seen():
    m = _model()
    (m(torch.randn(2, 12))).sum().backward()
    assert _trainer(m, FusedAdamW(m.parameters()), clip=1.0)._folds_clipping()
    assert not _trainer(m, torch.optim.AdamW(m.parameters()), clip=1.0)._folds_clipping()
    assert not _trainer(m, FusedAdamW(m[0].parameters()), clip=1.0)._folds_clipping()      # others keep scaled gradients
    hooked = FusedAdamW(m.parameters())
    hooked.register_step_pre_hook(lambda *a: None)
    assert not _trainer(m, hooked, clip=1.0)._folds_clipping()
    patched = FusedAdamW(m.parameters())
    patched.step = lambda: None
    assert not _trainer(m, patched, clip=1.0)._folds_clipping()


@pytest.mark.parametrize("make", [lambda p: FusedAdamW(p, lr=1e-2), lambda p: FusedSGD(p, lr=0.1)])
def test_parameters_outside_the_model_are_not_clipped(make):
    """An optimizer that also holds the criterion's parameter: clipping is that of the model's gradients alone."""

    class Scaled(torch.nn.Module):

        def __init__(self):
            super().__init__()
            self.scale = torch.nn.Parameter(torch.ones(1))

        def forward(self, out, target):
            return ((out * self.scale - target)**2).sum()

    a, b = _model(), _model()
    ca, cb = Scaled(), Scaled()
    oa, ob = (make(list(m.parameters()) + list(c.parameters())) for m, c in ((a, ca), (b, cb)))
    tr = Trainer(a, ca, oa, amp_dtype=None, clip=0.01, forward_fn=lambda m, x: (m(x["x"]), x["y"]))
    for i in range(3):
        g = torch.Generator().manual_seed(i)
        batch = dict(x=torch.randn(8, 12, generator=g), y=torch.randn(8, 3, generator=g))
        tr.step(batch)
        cb(b(batch["x"]), batch["y"]).backward()
        clip_grad_norm(list(b.parameters()), 0.01)
        ob.step()
        ob.zero_grad(set_to_none=True)
        for p, q in zip([*a.parameters(), ca.scale], [*b.parameters(), cb.scale]):
            assert torch.equal(p, q)
    # without a gradient it is not in the way
    (a(torch.randn(2, 12))).sum().backward()
    assert tr._folds_clipping()

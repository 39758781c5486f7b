"""Modules that ``torch.jit.trace`` records: the recorded module computes what the module does, on other inputs too."""
import types

import pytest
import torch


def _during_trace(f):
    got = []
    torch.jit.trace(lambda t: got.append(f()) or t * 2, (torch.ones(2), ), check_trace=False)
    return got[0]


def test_native_paths_stand_back_while_recorded(monkeypatch):
    from cubework_b200 import ops
    monkeypatch.setattr(ops.ext, "require", lambda: None)

    def on_gpu(*shape):                     # a stand-in with what the dispatch rules look at
        t = torch.zeros(*shape, dtype=torch.bfloat16)
        return types.SimpleNamespace(is_cuda=True, dtype=t.dtype, device=t.device, shape=t.shape, requires_grad=False,
                                     is_contiguous=lambda: True, data_ptr=lambda: 0, stride=t.stride, dim=t.dim)

    qkv, cache = on_gpu(2, 1, 3, 96), on_gpu(2, 3, 9, 32)
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda dev=None: True)
    rules = [lambda: ops._native(qkv, torch.bfloat16), lambda: ops.decode_ready(qkv, cache, cache, None),
             lambda: ops.prefill_ready(qkv, None)]
    for rule in rules:
        assert rule() and not _during_trace(rule)


def _traced(f, *examples):
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
        return torch.jit.trace(f, examples, check_trace=False)


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["linear", "norm", "attention"])
def test_traced_layer(which):
    from cubework_b200 import module as cube_nn
    from cubework_b200 import ops
    from cubework_b200.global_vars import env
    env.load(mode=None)
    torch.manual_seed(0)
    shape = (2, 40, 3, 96) if which == "attention" else (40, 64)
    a, b = (torch.randn(*shape, device="cuda").bfloat16() for _ in range(2))
    with torch.device("cuda"):
        f = {"linear": lambda: cube_nn.Linear(64, 72, activation="gelu"), "norm": lambda: cube_nn.LayerNorm(64),
             "attention": lambda: (lambda t: ops.attention_packed(t, True))}[which]()
    traced = _traced(f, a)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        for x in (b, a):
            assert torch.equal(traced(x), f(x))


@pytest.mark.gpu
def test_traced_cached_pass():
    """A prompt and one further token of OPT attention, recorded and replayed on other inputs."""
    from cubework_b200.global_vars import env
    from cubework_b200.models import opt
    env.load(mode=None)
    torch.manual_seed(0)
    m = opt.OPTAttention(64, 2).cuda().eval().requires_grad_(False)      # recorded as constants

    def prompt(x):
        o, (k, v) = m.forward_cached(x)
        return o, k, v

    def token(x, k, v):
        o, (k2, v2) = m.forward_cached(x, (k, v))
        return o, k2, v2

    x1, x2 = (torch.randn(2, 9, 64, device="cuda").bfloat16() for _ in range(2))
    t1, t2 = (torch.randn(2, 1, 64, device="cuda").bfloat16() for _ in range(2))
    traced = _traced(prompt, x1)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        past = prompt(x1)[1:]
        for got, ref in zip(traced(x2), prompt(x2)):      # the formulation rounds scores to 16 bits, the kernel does not
            assert (got.float() - ref.float()).norm() <= 0.03 * ref.float().norm()
    traced = _traced(token, t1, *past)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        for got, ref in zip(traced(t2, *past), token(t2, *past)):
            assert (got.float() - ref.float()).norm() <= 0.03 * ref.float().norm()

"""Transformer blocks as a caller sees them: the residual stream's type, hooks, and what recomputation keeps."""
import pytest
import torch

from cubework_b200.global_vars import env
from cubework_b200.models import opt, vit


def _vit_block(**kw):
    env.load(mode=None)
    torch.manual_seed(0)
    return vit.ViTBlock(32, 4, 64, **kw)


def _opt_layer(**kw):
    env.load(mode=None)
    torch.manual_seed(0)
    return opt.OPTDecoderLayer(32, 64, 4, dropout=0.0, **kw)


def _vit_formula(m, x):
    x = x + m.attn(m.norm1(x))
    return x + m.mlp(m.norm2(x))


def _opt_formula(m, x):
    x = x + m.self_attn(m.self_attn_layer_norm(x))
    return x + m.ffn(m.final_layer_norm(x))


@pytest.mark.parametrize("make,call,formula", [(_vit_block, lambda m, x: m(x), _vit_formula),
                                               (_opt_layer, lambda m, x: m(x)[0], _opt_formula)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_stream_keeps_its_type_under_autocast(make, call, formula, dtype):
    m, x = make(), torch.randn(2, 6, 32).to(dtype)
    with torch.autocast("cpu", dtype=torch.bfloat16):
        got, ref = call(m, x), formula(m, x)
    assert got.dtype == ref.dtype == dtype and torch.equal(got, ref)
    if dtype == torch.float32:
        got = call(m, x)
        assert got.dtype == dtype and torch.equal(got, formula(m, x))


def _vit_model(**kw):
    env.load(mode=None)
    torch.manual_seed(0)
    return vit.VisionTransformer(img_size=16, patch_size=8, num_classes=5, depth=3, hidden_size=32, num_heads=4,
                                 intermediate_size=64, dropout=0.0, **kw)


def _opt_model(**kw):
    env.load(mode=None)
    torch.manual_seed(0)
    return opt.OPT(vocab_size=64, hidden_size=32, num_hidden_layers=3, ffn_dim=64, num_attention_heads=4, dropout=0.0, init_std=0.1, **kw)


def _head_in(v):            # the zero-initialised head of a fresh ViT would hide everything before it
    torch.nn.init.normal_(v.head.dense.weight)
    return v


FAMILIES = {
    "vit": (lambda **kw: _head_in(_vit_model(**kw)), lambda: torch.randn(2, 3, 16, 16), lambda m: m.blocks, lambda m, x: m(x)),
    "opt": (_opt_model, lambda: torch.randint(2, 64, (2, 7)), lambda m: m.layers, lambda m, x: m(x)[0]),
}


def _streams(family, m, x):
    """The streams between the blocks, by the formulas, and the module's result."""
    got, formula = [], _vit_formula if family == "vit" else _opt_formula
    h = m.embed(x) if family == "vit" else m.embed_tokens(x) + m.embed_positions(torch.ones_like(x))
    for b in (m.blocks if family == "vit" else m.layers):
        h = formula(b, h)
        got.append(h)
    return got, m.head(m.norm(h)) if family == "vit" else m.lm_head(m.final_layer_norm(h))


@pytest.mark.parametrize("family", list(FAMILIES))
@pytest.mark.parametrize("which", ["block", "norm", "final norm", "global"])
def test_hooks_see_tensors(family, which):
    """Hooks on blocks and norms inside a model get the residual stream and its normalised value."""
    make, inputs, blocks, call = FAMILIES[family]
    m, x = make(), inputs()
    seen, handles = [], []
    keep = lambda mod, args, out: seen.append((mod, args, out))
    final = m.norm if family == "vit" else m.final_layer_norm
    first = blocks(m)[1].norm1 if family == "vit" else blocks(m)[1].self_attn_layer_norm
    second = blocks(m)[1].norm2 if family == "vit" else blocks(m)[1].final_layer_norm
    with torch.no_grad():
        streams, ref = _streams(family, m, x)
        plain = call(m, x)
        if which == "global":
            handles.append(torch.nn.modules.module.register_module_forward_hook(keep))
        else:
            for mod in {"block": list(blocks(m)), "norm": [first, second], "final norm": [final]}[which]:
                handles.append(mod.register_forward_hook(keep))
        out = call(m, x)
        for h in handles:
            h.remove()
    assert torch.equal(out, plain) and torch.equal(out, ref)
    watched = {mod: (args, res) for mod, args, res in seen}
    for i, b in enumerate(blocks(m)):
        if b in watched:
            args, res = watched[b]
            res = res if family == "vit" else res[0]
            assert torch.is_tensor(res) and torch.equal(res, streams[i])
            assert i == 0 or torch.equal(args[0], streams[i - 1])
            assert family == "opt" or len(args) == 1
    assert which == "norm" or which == "final norm" or all(b in watched for b in blocks(m))
    if first in watched:
        assert torch.equal(watched[first][0][0], streams[0]) and torch.equal(watched[first][1], first(streams[0]))
        assert torch.is_tensor(watched[second][1]) and len(watched[second][0]) == 1
    if final in watched:
        assert torch.equal(watched[final][0][0], streams[-1]) and torch.is_tensor(watched[final][1])


@pytest.mark.parametrize("family", list(FAMILIES))
def test_blocks_may_be_replaced(family):
    """Another module in a block's place (a wrapper, an identity) or an overridden forward is called as it always was."""

    class Wrapped(torch.nn.Module):

        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, h, *args):
            return self.inner(h, *args)

    class Skip(torch.nn.Module):

        def forward(self, h, *args):
            return h if family == "vit" else (h, None)

    make, inputs, blocks, call = FAMILIES[family]
    m, x = make(), inputs()
    with torch.no_grad():
        plain = call(m, x)
        b = blocks(m)
        b[1] = Wrapped(b[1])
        inner = b[2].forward
        b[2].forward = lambda h, *args: inner(h, *args)
        assert torch.equal(call(m, x), plain)
        b[1] = Skip()
        call(m, x)
        if family == "vit":
            m.norm = torch.nn.LayerNorm(32, eps=1e-6)
            b[0].norm2 = torch.nn.LayerNorm(32, eps=1e-6)
            call(m, x)


@pytest.mark.parametrize("family", list(FAMILIES))
def test_recomputed_blocks_keep_one_tensor(family):
    """With recomputation a block keeps its input for the backward pass and nothing else."""
    make, inputs, blocks, call = FAMILIES[family]
    kw = dict(checkpoint=True) if family == "vit" else dict(gradient_checkpointing=True)
    m, ref, x = make(**kw).train(), make().train(), inputs()
    ref.load_state_dict(m.state_dict())
    from cubework_b200.models.common import _Recompute
    kept, forward = [], _Recompute.forward

    def counted(ctx, fn, *args):
        kept.append(sum(torch.is_tensor(a) for a in args))
        return forward(ctx, fn, *args)

    _Recompute.forward = staticmethod(counted)
    try:
        out = call(m, x)
    finally:
        _Recompute.forward = staticmethod(forward)
    assert kept == [1] * len(blocks(m))
    out.square().sum().backward()
    r = call(ref, x)
    r.square().sum().backward()
    assert torch.equal(out, r)
    for (n, p), q in zip(m.named_parameters(), ref.parameters()):
        assert torch.allclose(p.grad, q.grad, rtol=1e-4, atol=1e-6 * q.grad.abs().max().item()), n


def test_cached_attention_reads_the_first_two_entries():
    """A cache entry may carry more than keys and values."""
    env.load(mode=None)
    torch.manual_seed(0)
    m = opt.OPTAttention(32, 4)
    x, t = torch.randn(2, 5, 32), torch.randn(2, 1, 32)
    with torch.no_grad():
        k, v = m.forward_cached(x)[1]
        ref = m.forward_cached(t, (k, v))[0]
        assert torch.equal(m.forward_cached(t, (k, v, "a note"))[0], ref)

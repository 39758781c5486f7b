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

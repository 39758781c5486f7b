"""The native autograd nodes against the Python functions they stand in for, and where those have to stay."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grads(out, inputs, seeds):
    outs = out if isinstance(out, (tuple, list)) else [out]
    return torch.autograd.grad(outs, inputs, seeds, allow_unused=True)


def _close(a, b):
    assert (a is None) == (b is None)
    if a is not None:      # the same kernels; only the order of split fp32 sums may differ
        assert a.dtype == b.dtype and a.shape == b.shape
        assert (a.double() - b.double()).norm() <= 1e-5 * b.double().norm() + 1e-12


@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act,bias,out_in,strided", [(None, True, True, False), ("gelu", True, True, True), ("relu", False, True, False),
                                                     (None, False, False, True)])
def test_linear(params, x_dtype, act, bias, out_in, strided):
    from cubework_b200 import ops
    from cubework_b200.parallel.functional import _LocalLinear
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(2, 40, 72, generator=g, device="cuda").to(x_dtype)
    x = (x[:, ::2] if strided else x[:, :20]).detach().requires_grad_(True)
    w = torch.randn(*((104, 72) if out_in else (72, 104)), generator=g, device="cuda").to(params).requires_grad_(True)
    b = torch.randn(104, generator=g, device="cuda").to(params).requires_grad_(True) if bias else None
    inputs = [t for t in (x, w, b) if t is not None]
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = ops.native_linear(x, w, b, out_in, act)
        ref = _LocalLinear.apply(x, w, b, out_in, act, True)
    assert y is not None and torch.equal(y, ref)
    dy = torch.randn(ref.shape, generator=g, device="cuda").to(ref.dtype)
    for a, r in zip(_grads(y, inputs, [dy]), _grads(ref, inputs, [dy])):
        _close(a, r)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert torch.equal(ops.native_linear(x, w, b, out_in, act), ref)


@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,H", [(3, 64), (700, 1600), (10, 2056)])
def test_norm(params, rows, H):
    from cubework_b200 import ops
    from cubework_b200.parallel.functional import _AddLayerNorm, _LayerNorm
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, r = (torch.randn(rows, H, generator=g, device="cuda").bfloat16().requires_grad_(True) for _ in range(2))
    gamma, beta = (torch.randn(H, generator=g, device="cuda").to(params).requires_grad_(True) for _ in range(2))
    seeds = [torch.randn(rows, H, generator=g, device="cuda").bfloat16() for _ in range(2)]
    got, ref = ops.native_norm(x, r, gamma, beta, 1e-5), _AddLayerNorm.apply(x, r, gamma, beta, 1e-5)
    assert all(torch.equal(a, b) for a, b in zip(got, ref))
    for a, b in zip(_grads(got, [x, r, gamma, beta], seeds), _grads(ref, [x, r, gamma, beta], seeds)):
        _close(a, b)
    got, ref = ops.native_norm(x, None, gamma, beta, 1e-5), _LayerNorm.apply(x, gamma, beta, 1e-5)
    assert torch.equal(got[0], ref)
    for a, b in zip(_grads(got, [x, gamma, beta], seeds[:1]), _grads(ref, [x, gamma, beta], seeds[:1])):
        _close(a, b)
    # a gradient for only one of the two outputs
    s, y = ops.native_norm(x, r, gamma, beta, 1e-5)
    rs, ry = _AddLayerNorm.apply(x, r, gamma, beta, 1e-5)
    _close(_grads(s, [x], seeds[:1])[0], _grads(rs, [x], seeds[:1])[0])


def test_where_the_python_functions_stay():
    from cubework_b200 import ops
    from cubework_b200.parallel.functional import layer_norm, local_linear
    x = torch.randn(4, 64, device="cuda").bfloat16()
    w = torch.randn(32, 64, device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert ops.native_linear(x, torch.randn(30, 64, device="cuda"), None, True, None) is None       # padded extents
        assert ops.native_linear(x, w.half(), None, True, None) is None                                 # another 16-bit type
        swapped = w.clone()
        swapped.storage_is_swapped = True
        assert ops.native_linear(x, swapped, None, True, None) is None
    assert ops.native_linear(x.float(), w, None, True, None) is None                                    # fp32 compute
    assert ops.native_norm(x.float(), None, torch.ones(64, device="cuda"), torch.zeros(64, device="cuda"), 1e-5) is None
    ones, zeros = torch.ones(64, device="cuda"), torch.zeros(64, device="cuda")
    for f in (lambda t: local_linear(t, w.bfloat16()).float().sum(), lambda t: layer_norm(t, ones, zeros, 1e-5).float().sum()):
        with pytest.raises(RuntimeError):
            torch.func.grad(f)(x)                # refused before, refused still


def test_saved_tensor_hooks_see_what_is_kept():
    from cubework_b200.parallel.functional import local_linear
    x = torch.randn(4, 64, device="cuda").bfloat16().requires_grad_(True)
    w = torch.randn(32, 64, device="cuda", requires_grad=True)
    seen = []
    with torch.autocast("cuda", dtype=torch.bfloat16), \
            torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        y = local_linear(x, w, None, True, "relu")
    assert len(seen) >= 3
    y.float().sum().backward()
    assert x.grad is not None and w.grad is not None


@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
def test_saved_tensor_hooks_see_the_same_tensors(params):
    """What is offered to hooks (offloading) is what the Python functions offer, and not the weight's 16-bit copy besides."""
    from cubework_b200 import ops
    from cubework_b200.parallel.functional import _AddLayerNorm, _LocalLinear
    x = torch.randn(24, 64, device="cuda").bfloat16().requires_grad_(True)
    w, b = torch.randn(32, 64, device="cuda").to(params).requires_grad_(True), torch.zeros(32, device="cuda", dtype=params)
    gamma = torch.ones(64, device="cuda", dtype=params)
    qkv = torch.randn(2, 40, 3, 96, device="cuda").bfloat16().requires_grad_(True)

    def offered(f):
        seen = []
        with torch.autocast("cuda", dtype=torch.bfloat16), \
                torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append((tuple(t.shape), t.dtype)) or t, lambda t: t):
            f()
        return sorted((s, str(d)) for s, d in seen if 0 not in s)

    assert offered(lambda: ops.native_linear(x, w, b, True, "relu")) == offered(lambda: _LocalLinear.apply(x, w, b, True, "relu", True))
    assert offered(lambda: ops.native_linear(x, w, b, True, None)) == offered(lambda: _LocalLinear.apply(x, w, b, True, None, True))
    assert offered(lambda: ops.native_norm(x, x, gamma, gamma, 1e-5)) == offered(lambda: _AddLayerNorm.apply(x, x, gamma, gamma, 1e-5))
    assert offered(lambda: ops.attention_packed(qkv, True)) == offered(lambda: ops._AttentionFn.apply(qkv, True, None, 0.1))

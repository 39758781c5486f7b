"""Cached decoding on the GPU: the fused append + attention kernel and the weight-streaming GEMM of a few rows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

UNIT = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}     # largest relative error of one rounding (8 / 11 significant bits)


def _ops():
    from cubework_b200 import ops
    return ops


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,T,dh,padded,strided", [
    (1, 1, 1, 8, False, False),         # one key in the cache, the narrowest head
    (2, 3, 31, 48, True, False),        # idle lanes of a key group
    (1, 16, 101, 48, False, True),      # the cache as a prompt leaves it: views of the packed projection
    (8, 32, 1000, 64, True, False),
    (3, 5, 128, 80, True, True),
    (2, 4, 1023, 128, True, False),
    (1, 2, 300, 256, False, False),     # a whole warp per key, the widest head
])
def test_decode_attention(dtype, B, H, T, dh, padded, strided):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    qkv = torch.randn(B, 1, H, 3 * dh, generator=g, device="cuda").to(dtype)
    if strided:
        past = torch.randn(B, T, H, 3 * dh, generator=g, device="cuda").to(dtype).permute(0, 2, 1, 3)
        k, v = past[..., dh:2 * dh], past[..., 2 * dh:]
    else:
        k, v = (torch.randn(B, H, T, dh, generator=g, device="cuda").to(dtype) for _ in range(2))
    bias = None
    if padded:
        bias = torch.zeros(B, T + 1, device="cuda")
        bias[:, :T // 3] = -10000.0
        bias[0, 0] = -math.inf          # a dropped key
    assert ops.decode_ready(qkv, k, v, bias)
    out, k2, v2 = ops.decode_attention(qkv, k, v, bias)
    q, kn, vn = qkv.permute(0, 2, 1, 3).chunk(3, dim=-1)
    want_k, want_v = torch.cat([k, kn], 2), torch.cat([v, vn], 2)
    assert torch.equal(k2, want_k) and torch.equal(v2, want_v) and k2.is_contiguous() and v2.is_contiguous()
    s = (q.double() @ want_k.double().transpose(-1, -2)) / math.sqrt(dh)
    if bias is not None:
        s = s + bias.double()[:, None, None, :]
    ref = (torch.softmax(s, -1) @ want_v.double()).transpose(1, 2).reshape(B, 1, H * dh)
    # one rounding of a value of at most max|v|, and fp32 sums; a bias of -1e4 leaves 2^-10 of absolute score, on keys
    # whose weight is zero unless all are dropped
    bound = UNIT[dtype] * ref.abs() + 1e-4 * want_v.double().abs().max()
    assert ((out.double() - ref).abs() <= bound).all()


def test_decode_attention_all_keys_dropped():
    """No key with a finite score: NaN, as the softmax of such a row."""
    ops = _ops()
    qkv = torch.randn(1, 1, 2, 96, device="cuda").bfloat16()
    k = torch.randn(1, 2, 40, 32, device="cuda").bfloat16()
    out = ops.decode_attention(qkv, k, k, torch.full((1, 41), -math.inf, device="cuda"))[0]
    assert out.isnan().all()


def test_decode_ready_refuses():
    ops = _ops()
    qkv = torch.randn(2, 1, 2, 96, device="cuda").bfloat16()
    k = torch.randn(2, 2, 9, 32, device="cuda").bfloat16()
    assert ops.decode_ready(qkv, k, k, None)
    assert not ops.decode_ready(qkv, k.half(), k, None)                                  # another dtype
    assert not ops.decode_ready(qkv, k, k[:, :, :8], None)                               # lengths differ
    assert not ops.decode_ready(qkv, k.transpose(-1, -2).contiguous().transpose(-1, -2), k, None)
    assert not ops.decode_ready(qkv, k, k, torch.zeros(1, 10, device="cuda"))            # a bias that broadcasts
    assert not ops.decode_ready(qkv.expand(2, 3, 2, 96), k, k, None)                     # several query tokens
    assert not ops.decode_ready(qkv.clone().requires_grad_(True), k, k, None)
    odd = torch.empty(k.numel() + 1, device="cuda", dtype=k.dtype)[1:].view_as(k)        # rows at odd addresses
    assert not ops.decode_ready(qkv, odd, k, None)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,act", [
    (1, 1, 8, None), (1, 768, 768, "relu"), (8, 2048, 2048, None), (9, 2304, 768, "gelu"), (16, 50, 4104, None),
    (17, 2048, 8192, "relu"), (32, 1000, 520, "gelu"), (33, 1000, 520, "gelu"), (3, 250, 1001, None),
    (16, 2368, 264, None), (16, 2376, 264, "relu"), (32, 4736, 264, "gelu"), (32, 4744, 264, None),      # ends of the rule for the warps
    (17, 9472, 136, None), (17, 9480, 136, "relu"),                                                       # ... and for the kernel
    (9, 16392, 2048, None), (9, 16392, 2056, "gelu"), (8, 20488, 1024, None), (8, 20488, 1016, "relu"),
    (9, 16392, 1024, None), (8, 4744, 8192, "relu"), (5, 7112, 8192, None), (32, 4744, 8192, "gelu"),
])
def test_skinny_gemm(dtype, M, N, K, act):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(M * 100 + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(dtype)
    b = torch.randn(N, generator=g, device="cuda")
    streams = M <= 32 and (M <= 16 or N <= 9472) and (M <= 8 or M > 16 or N <= 16384 or 1024 < K <= 2048) and \
        (M > 8 or N <= 20480 or 1024 <= K <= 8192)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (ops.ext.require().gemm_route(M, N, K, False, True, act or "", False, True) == -1) == streams
    y, z = ops.gemm(x, w, trans_b=True, bias=b, act=act, pre_act_out=True)
    ref = x.double() @ w.double().t() + b.double()
    # one rounding of the result, and fp32 sums of K products of unit variance / K
    tol = lambda t: UNIT[dtype] * t.abs() + 1e-5 * math.sqrt(K) + 1e-6
    assert ((z.double() - ref).abs() <= tol(ref)).all()
    out = torch.nn.functional.gelu(ref) if act == "gelu" else ref.relu() if act == "relu" else ref
    assert ((y.double() - out).abs() <= tol(out)).all()


@pytest.mark.parametrize("params,pad", [("master", True), ("16bit", False)])
def test_opt_cached_pass_matches_the_formulation(params, pad):
    """Prompt and two further tokens through the kernels against the same passes in fp32 PyTorch (CPU)."""
    import contextlib

    from cubework_b200.global_vars import env
    from cubework_b200.models import opt
    env.load(mode=None)
    torch.manual_seed(0)
    m = opt.OPT(vocab_size=512, hidden_size=128, num_hidden_layers=2, ffn_dim=512, num_attention_heads=2, dropout=0.0,
                max_position_embeddings=256, init_std=0.05, dtype=torch.bfloat16 if params == "16bit" else None).eval()
    host = opt.OPT(vocab_size=512, hidden_size=128, num_hidden_layers=2, ffn_dim=512, num_attention_heads=2, dropout=0.0,
                   max_position_embeddings=256).eval()
    host.load_state_dict({k: v.float() for k, v in m.state_dict().items()})
    m.cuda()
    cast = (lambda: torch.autocast("cuda", dtype=torch.bfloat16)) if params == "master" else contextlib.nullcontext
    ids = torch.randint(2, 512, (2, 37))
    mask = torch.ones(2, 37)
    if pad:
        mask[1, :9] = 0
    past = hpast = None
    with torch.no_grad(), cast():
        for _ in range(3):
            logits, past = m(ids.cuda(), mask.cuda(), past_key_values=past, use_cache=True)
            with torch.autocast("cuda", enabled=False):
                hlogits, hpast = host(ids, mask, past_key_values=hpast, use_cache=True)
            keep = mask[:, -ids.shape[1]:].bool()
            err = (logits.float().cpu() - hlogits)[keep].norm() / hlogits[keep].norm()
            assert err < 0.03, err          # two layers of bf16 roundings (2^-9 each, a dozen of them)
            ids, mask = torch.randint(2, 512, (2, 1)), torch.cat([mask, torch.ones(2, 1)], 1)

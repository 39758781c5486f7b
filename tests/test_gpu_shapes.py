"""Kernels at the edges of their tiles and dispatch rules: column sums over few and many columns, wide layer norms with a
residual, the row sums and the dQ conversion of attention, wide heads, and the GEMM on pairs of SMs."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

UNIT = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}     # largest relative error of one rounding (8 / 11 significant bits)

SUM_DEPTH = 64


def _ops():
    from cubework_b200 import ops
    from cubework_b200.ops import ext
    ext.require()
    return ops, ext


@pytest.mark.parametrize("act", ["gelu", "relu", None])
@pytest.mark.parametrize("M,N", [(1, 8), (3, 264), (17, 768), (1000, 1600), (513, 3072), (40, 6400), (5000, 2056)])
def test_act_backward_stripes(M, N, act):
    ops, _ = _ops()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    dy = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    if act is None:
        got, ref = ops.column_sum(dy), dy.double().sum(0)
    else:
        z = torch.randn(M, N, generator=g, device="cuda").bfloat16()
        zz = z.double().requires_grad_(True)
        (torch.nn.functional.gelu(zz) if act == "gelu" else zz.relu()).backward(dy.double())
        dz, got = ops.act_backward(dy, z, act, want_bias_grad=True)
        # one rounding, and the error function's 1.5e-7 times |dy|
        assert ((dz.double() - zz.grad).abs() <= UNIT[torch.bfloat16] * zz.grad.abs() + 1e-5).all()
        ref = dz.double().sum(0)
    # of the rounded gradients.  Fewer than 64 additions lie between a term and the result (rows of a thread, row groups, partial
    # sums), each of which rounds a partial sum of the magnitudes at most: a row that is lost or taken twice shows
    terms = dy if act is None else dz
    assert ((got.double() - ref).abs() <= SUM_DEPTH * 2.0**-24 * terms.double().abs().sum(0) + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,H", [(1, 8), (1, 2056), (300, 4096), (1200, 5120), (5, 6144), (7, 8200), (3, 16384),
                                    (700, 1280), (297, 1288), (700, 1536), (700, 1544), (2000, 2048)])   # ends of the rules
def test_wide_layer_norm_with_residual(rows, H, dtype):
    ops, _ = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x, r, dy, ds = (torch.randn(rows, H, generator=g, device="cuda").to(dtype) for _ in range(4))
    flat = torch.randn(2 * H + 1, generator=g, device="cuda")
    gamma, beta = flat[1:H + 1], flat[H + 1:]                      # views that start 4 bytes off a 16-byte boundary
    y, mean, rstd, total = ops.layer_norm_fwd(x, gamma, beta, 1e-5, residual=r)
    assert torch.equal(total, x + r)
    t = total.double().requires_grad_(True)
    gd, bd = gamma.double().requires_grad_(True), beta.double().requires_grad_(True)
    ref = torch.nn.functional.layer_norm(t, (H, ), gd, bd, 1e-5)
    ref.backward(dy.double())
    assert ((y.double() - ref).abs() <= UNIT[dtype] * ref.abs() + 1e-5).all()
    dx, dg, db = ops.layer_norm_bwd(dy, total, mean, rstd, gamma, dres=ds)
    want = t.grad + ds.double()
    assert ((dx.double() - want).abs() <= UNIT[dtype] * want.abs() + 1e-5).all()
    # sums over the rows as above; a normalised value carries a few roundings of its own (mean, deviation, their product)
    xhat = (t.detach() - t.detach().mean(1, keepdim=True)) * (t.detach().var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    for got, want, terms in ((dg, gd.grad, dy.double() * (xhat.abs() + 1)), (db, bd.grad, dy.double())):
        assert ((got.double() - want).abs() <= (SUM_DEPTH + 16) * 2.0**-24 * terms.abs().sum(0) + 1e-6).all()
    y2, _, _ = ops.layer_norm_fwd(total, gamma, beta, 1e-5)       # may sum in another order (another kernel)
    assert ((y2.double() - ref).abs() <= UNIT[dtype] * ref.abs() + 1e-5).all()


@pytest.mark.parametrize("H", [1280, 1288, 2048, 4096])           # both kernels of the backward
def test_layer_norm_refuses_parameters_of_another_length(H):
    ops, _ = _ops()
    x, r = (torch.randn(4, H, device="cuda").bfloat16() for _ in range(2))
    ones = torch.ones(H, device="cuda")
    y, mean, rstd, total = ops.layer_norm_fwd(x, ones, ones, 1e-5, residual=r)
    for bad in (ones[:H - 8], torch.ones(H + 8, device="cuda")):
        for dres in (None, r):
            with pytest.raises(RuntimeError, match="norm parameters"):
                ops.layer_norm_bwd(y, total, mean, rstd, bad, dres=dres)
        with pytest.raises(RuntimeError, match="norm parameters"):
            ops.layer_norm_fwd(x, bad, ones, 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,dh,causal,pad", [
    (1, 1, 1, 80, True, False),          # one row of one tile
    (1, 128, 3, 128, True, False),       # one full tile, its neighbour does not exist
    (2, 129, 2, 128, True, True),        # one row in the second tile
    (1, 257, 4, 72, False, False),       # an odd number of tiles, no mask
    (2, 640, 5, 96, True, True),         # more key blocks than ring stages
    (3, 300, 2, 100, True, False),       # a head dim that needs the padded copy
    (2, 197, 3, 48, False, False),       # the vector row sums with idle lanes
    (2, 70, 3, 24, True, False),         # ... and with four lanes
    (4, 900, 40, 128, True, True),       # several items per CTA
    (3, 100, 5, 32, True, True),         # one tile per head, fewer than there are SMs
    (41, 100, 11, 25, True, True),       # ... and more, an odd number: the last has no partner
    (31, 100, 11, 48, True, True),
    (30, 128, 12, 80, False, True),
    (20, 300, 16, 64, False, True),      # an odd last tile alone, then neighbours
    (10, 300, 17, 25, True, True),       # odd last tiles of two heads, then neighbours
    (10, 300, 17, 96, False, True),
    (2, 640, 5, 48, True, True),
])
def test_attention_tiles(dtype, B, T, H, dh, causal, pad):
    ops, ext = _ops()
    g = torch.Generator(device="cuda").manual_seed(B * T + dh)
    qkv = torch.randn(B, T, H, 3 * dh, generator=g, device="cuda")
    qkv[..., :dh] *= 3.0                                          # scores that make the running maximum move
    qkv = qkv.to(dtype).requires_grad_(True)
    bias = None
    if pad:
        bias = torch.zeros(B, T, device="cuda")
        bias[-1, T // 2:] = -10000.0
        bias[::3, :T // 5] = -1.5                                 # another bias for every third sequence
    dout = torch.randn(B, T, H * dh, generator=g, device="cuda").to(dtype)
    out = ops.attention_packed(qkv, causal, bias)
    out.backward(dout)
    ext.check_status()
    ref_in = qkv.detach().float().requires_grad_(True)
    q, k, v = ref_in.permute(0, 2, 1, 3).chunk(3, dim=-1)
    ref = ops.attention_reference(q, k, v, causal, bias).transpose(1, 2).reshape(B, T, H * dh)
    ref.backward(dout.float())
    # probabilities and results rounded to 16 bits; gradients pass two such products more
    tol = 4 * UNIT[dtype]
    assert (out.float() - ref).norm() <= tol * ref.norm()
    assert (qkv.grad.float() - ref_in.grad).norm() <= 2 * tol * ref_in.grad.norm()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K,pairs,pairs32", [       # whether 16-bit and fp32 outputs go to the kernel on pairs
    (256, 256, 64, False, False),         # one tile, one k-block
    (264, 64, 72, False, False),
    (1000, 1608, 200, False, False),
    (33, 50304, 136, False, False),
    (333, 10240, 2056, False, False),     # one wave of single CTAs, two of pairs
    (256, 256, 8128, False, False),       # one k-block less than the rule asks for
    (256, 256, 8192, True, False),        # one tile
    (264, 136, 8200, True, False),        # a second row block of 8 rows, the narrowest tile, a ragged last k-block
    (1000, 1608, 8200, True, True),       # ragged in every extent; split K
    (4096, 1600, 2600, True, True),       # two waves, a last tile of 64 columns
    (2048, 776, 8200, True, True),        # one wave of long tiles
    (136, 50304, 1544, True, True),       # almost half of every row block empty, several tiles per pair
    (4096, 8192, 776, True, True),        # short tiles in many waves
])
def test_gemm_on_pairs(dtype, trans_a, trans_b, M, N, K, pairs, pairs32):
    ops, ext = _ops()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    pad = lambda n: (n + 7) // 8 * 8
    M = pad(M) if trans_a else M
    a = torch.randn((K, M) if trans_a else (M, K), generator=g, device="cuda").to(dtype)
    b = torch.randn((N, K) if trans_b else (K, N), generator=g, device="cuda").to(dtype)
    route = ext.require().gemm_route
    assert (route(M, N, K, trans_a, True, "", False, False) > 0) == pairs and (route(M, N, K, trans_a, trans_b, "", True, False) > 0) == pairs32
    assert not pairs or route(M, N, K, trans_a, trans_b, "", False, False) > 0
    ref = (a.float().t() if trans_a else a.float()) @ (b.float().t() if trans_b else b.float())
    out32 = ops.gemm(a, b, trans_a, trans_b, out_dtype=torch.float32)
    out = ops.gemm(a, b, trans_a, trans_b)
    ext.check_status()
    assert (out32 - ref).norm() <= 1e-5 * ref.norm()              # both sums are fp32
    assert ((out.float() - ref).abs() <= UNIT[dtype] * ref.abs() + 1e-4 * math.sqrt(K)).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", [None, "gelu", "relu"])
@pytest.mark.parametrize("M,N,K", [
    (300, 1600, 264), (520, 1000, 264), (4096, 160, 264), (700, 2300, 264), (260, 60, 264),      # the single-CTA kernel
    (300, 1600, 8200),             # one live chunk of 64 columns in the last tile, rows for only half of a cluster
    (520, 1000, 8200),             # a half chunk at the matrix's end
    (4096, 160, 8200),             # one tile wide, three chunks of which the last is half
    (700, 2300, 8200),             # a row pitch that TMA cannot store
    (260, 132, 8200),              # ... with one row quarter of four rows and a chunk of four columns
    (256, 260, 8200),              # ... with a last tile of four columns
    (6304, 1544, 1544),            # several tiles per pair: both accumulators and their hand-over
])
def test_gemm_on_pairs_epilogue(M, N, K, act, dtype):
    """Bias, activation and the pre-activation copy: whole chunks, half chunks at a tile's or the matrix's end, and a row
    pitch that TMA cannot store, in the kernel for pairs of SMs and in the one for single CTAs."""
    ops, ext = _ops()
    route = ext.require().gemm_route
    assert all((route(M, N, K, False, True, act or "", False, z) > 0) == (K != 264) for z in (False, True))
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    b = (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(dtype)
    bias = torch.randn(N, generator=g, device="cuda")
    z_ref = a.double() @ b.double().t() + bias.double()
    y_ref = torch.nn.functional.gelu(z_ref) if act == "gelu" else z_ref.relu() if act == "relu" else z_ref
    y, z = ext.gemm(a, b, False, True, bias, act, dtype, True)
    y1 = ext.gemm(a, b, False, True, bias, act, dtype, False)
    y32 = ext.gemm(a, b, False, True, bias, act, torch.float32, False)
    ext.check_status()
    # K / 16 accumulations, each rounding a running sum below 8 to 24 bits, and the activation's error
    u, acc = UNIT[dtype], K / 16 * 2.0**-24 * 8 + 1e-5
    assert ((z.double() - z_ref).abs() <= u * z_ref.abs() + acc).all()
    assert ((y.double() - y_ref).abs() <= u * y_ref.abs() + acc).all() and torch.equal(y, y1)
    assert ((y32.double() - y_ref).abs() <= acc).all()

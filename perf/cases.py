"""Workloads that stand for what a user has the framework do, with their sizes, inputs, work and tolerances.

Seven kinds, all on one device and through the public entry points (``models``, ``module``, ``engine``, ``optim``):

* ``gpt2`` / ``vit`` / ``opt``  one optimisation step (``Trainer.step``: forward, loss, backward, clipping, AdamW) of a stack
                       of the presets' widths.  Depth is at most four layers, so that the weights come back one by one;
                       deeper models repeat the same layer.  Outputs: the loss and every updated weight.  GPT-2 stacks of up
                       to two layers also return the first moments (0.1 x the gradient after one step).
* ``linear``           forward + backward of one ``module.Linear``, as in ``benchmark/linear``.
* ``eval``             ``Trainer.evaluate``: logits and loss of a whole model.
* ``prefill``/``decode``  OPT with a key/value cache: a prompt at once, then one more token.

Sizes are the ones of the presets, of the benchmark drivers and of the tests.  ``draw`` mixes them over the whole
range, with odd sequence lengths, batches and feature counts.
"""
import contextlib
import math

import torch

from cubework_b200 import module as cube_nn
from cubework_b200.engine import Trainer
from cubework_b200.global_vars import env
from cubework_b200.models import gpt2, opt, vit
from cubework_b200.optim import FusedAdamW

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
VOCAB = 50304


def listed():
    return [
        # the smallest configuration (2 layers, hidden 128, sequence 64, batch 4): a step of launches and host work
        dict(name="gpt2_tiny_step", kind="gpt2", hidden=128, heads=4, depth=2, vocab=1024, batch=4, seq=64, dtype="bf16",
             ckpt=False, pad=False),
        # the headline training step: GPT-2 XL layers (64 heads x 25), batch 32 x 1024 tokens
        dict(name="gpt2_xl_step", kind="gpt2", hidden=1600, heads=64, depth=4, vocab=VOCAB, batch=32, seq=1024, dtype="bf16",
             ckpt=False, pad=False),
        # fp16 with a loss scaler, recomputed blocks, padded sequences of a length that is no multiple of a tile
        dict(name="gpt2_medium_fp16_ckpt", kind="gpt2", hidden=1024, heads=16, depth=2, vocab=VOCAB, batch=8, seq=1000,
             dtype="fp16", ckpt=True, pad=True),
        # ViT-B/16 layers at the benchmark's global batch: 197 tokens per image, no causal mask
        dict(name="vit_base_step", kind="vit", hidden=768, heads=12, depth=4, img=224, patch=16, classes=1000, batch=256,
             dtype="bf16"),
        # OPT-13B layers (40 heads x 128, ReLU) at sequence 2048 with recomputed blocks
        dict(name="opt_13b_step", kind="opt", hidden=5120, heads=40, depth=2, vocab=50272, batch=4, seq=2048, dtype="bf16",
             ckpt=True, pad=False),
        # a small batch of OPT-125M layers with ragged, padded sequences
        dict(name="opt_125m_step_ragged", kind="opt", hidden=768, heads=16, depth=4, vocab=VOCAB, batch=3, seq=333,
             dtype="bf16", ckpt=False, pad=True),
        # the parallel-linear microbenchmark (16384 rows, K = N = 8192)
        dict(name="linear_8192", kind="linear", rows=16384, fan_in=8192, fan_out=8192, act="", dtype="bf16"),
        # the first MLP linear of ViT-B on 32 images, with its fused activation
        dict(name="linear_fc1_gelu", kind="linear", rows=6304, fan_in=768, fan_out=3072, act="gelu", dtype="bf16"),
        # a test pass of the whole ViT-B (16 heads x 48) on the last, incomplete batch
        dict(name="vit_base_eval", kind="eval", family="vit", hidden=768, heads=16, depth=12, img=224, patch=16, classes=1000,
             batch=100, dtype="bf16"),
        # OPT-1.3B: four prompts of 500 tokens into the cache, fp32 masters under autocast
        dict(name="opt_1b_prefill", kind="prefill", hidden=2048, heads=32, depth=24, batch=4, seq=500, params="master", pad=False),
        # OPT-1.3B: one more token for eight left-padded requests
        dict(name="opt_1b_decode", kind="decode", hidden=2048, heads=32, depth=24, batch=8, seq=1000, params="master", pad=True),
        # OPT-125M: one more token for one request, 16-bit parameters
        dict(name="opt_125m_decode", kind="decode", hidden=768, heads=16, depth=12, batch=1, seq=100, params="16bit", pad=False),
    ]


# ------------------------------------------------------------------------------------------------------ drawn cases
MOST_FLOPS = 4.0e13       # a drawn case costs no more than the largest listed one
GPT2_WIDTHS = [(128, 4), (768, 16), (1024, 16), (1280, 20), (1600, 64), (1600, 25), (2880, 64), (4096, 64)]
VIT_WIDTHS = [(384, 16, 16), (768, 12, 16), (768, 16, 16), (1024, 16, 16), (1280, 16, 14)]
OPT_WIDTHS = [(768, 16), (1024, 16), (2048, 32), (2560, 32), (4096, 64), (5120, 40), (5120, 64)]
CACHE_MODELS = [(768, 16, 12), (1024, 16, 24), (2048, 32, 24)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _features(rng):
    n = _log_int(rng, 512, 12288)
    return n if rng.random() < 0.15 else max(8, n // 8 * 8)      # now and then no multiple of eight


def _smaller(case):
    """Halve the batch (or the rows) until the case is no larger than the largest listed one."""
    key = "rows" if case["kind"] == "linear" else "batch"
    while work(case)["flops"] > MOST_FLOPS and case[key] > 1:
        case[key] //= 2
    return case


def draw(rng):
    kind = rng.choice(["gpt2", "gpt2", "vit", "opt", "linear", "linear", "eval", "prefill", "decode", "decode"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if kind == "gpt2":
        hidden, heads = rng.choice(GPT2_WIDTHS)
        tiny = hidden == 128
        seq = _log_int(rng, 33, 128) if tiny else _log_int(rng, 64, 1024)
        return _smaller(dict(kind=kind, hidden=hidden, heads=heads, depth=rng.randint(1, 4), vocab=1024 if tiny else VOCAB,
                             batch=min(_log_int(rng, 1, 64), 32768 // seq), seq=seq, dtype=dtype, ckpt=rng.random() < 0.4,
                             pad=rng.random() < 0.4))
    if kind == "vit":
        hidden, heads, patch = rng.choice(VIT_WIDTHS)
        return _smaller(dict(kind=kind, hidden=hidden, heads=heads, depth=rng.randint(1, 4), img=224, patch=patch, classes=1000,
                             batch=_log_int(rng, 8, 256), dtype=dtype))
    if kind == "opt":
        hidden, heads = rng.choice(OPT_WIDTHS)
        seq = _log_int(rng, 128, 2048)
        return _smaller(dict(kind=kind, hidden=hidden, heads=heads, depth=rng.randint(1, 2 if hidden > 2048 else 4), vocab=50272,
                             batch=min(_log_int(rng, 1, 16), 16384 // seq), seq=seq, dtype=dtype, ckpt=rng.random() < 0.6,
                             pad=rng.random() < 0.4))
    if kind == "linear":
        return _smaller(dict(kind=kind, rows=_log_int(rng, 64, 16384), fan_in=_features(rng), fan_out=_features(rng),
                             act=rng.choice(["", "", "gelu", "relu"]), dtype=dtype))
    if kind == "eval":
        family = rng.choice(["gpt2", "vit", "opt"])
        if family == "vit":
            hidden, heads, patch = rng.choice(VIT_WIDTHS)
            return _smaller(dict(kind=kind, family=family, hidden=hidden, heads=heads, depth=12, img=224, patch=patch,
                                 classes=1000, batch=_log_int(rng, 1, 128), dtype=dtype))
        hidden, heads = rng.choice([(768, 16), (1024, 16), (1280, 20), (1600, 64)] if family == "gpt2" else OPT_WIDTHS[:3])
        seq = _log_int(rng, 64, 1024)
        return _smaller(dict(kind=kind, family=family, hidden=hidden, heads=heads, depth=12, vocab=VOCAB,
                             batch=min(_log_int(rng, 1, 16), 8192 // seq), seq=seq, dtype=dtype, pad=rng.random() < 0.5))
    hidden, heads, depth = rng.choice(CACHE_MODELS)
    case = dict(kind=kind, hidden=hidden, heads=heads, depth=depth, params=rng.choice(["master", "16bit"]),
                pad=rng.random() < 0.5)
    if kind == "prefill":
        seq = _log_int(rng, 16, 1024)
        return dict(case, batch=min(_log_int(rng, 1, 8), 4096 // seq), seq=seq)
    return dict(case, batch=_log_int(rng, 1, 16), seq=_log_int(rng, 16, 1024))


# ------------------------------------------------------------------------------------------------------ preparation
def _settle(model):
    """Biases and norm scales as a trained model has them, not the zeros and ones of the first step."""
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() == 1:
                p.normal_(0.0, 0.1)
                if "norm" in name and name.endswith("weight"):
                    p.add_(1.0)
            elif name.endswith(("cls_token", "pos_embed")) or "head" in name:
                p.normal_(0.0, 0.02)
    return model


def _family(case):
    return case.get("family", case["kind"] if case["kind"] in ("gpt2", "vit") else "opt")


def _mask(case, gen, left=False):
    """1 / 0 mask ``[batch, seq]``: all ones, or with up to a third of each sequence but the first padded."""
    batch, seq = case["batch"], case["seq"]
    mask = torch.ones(batch, seq, device="cuda")
    if case["pad"]:
        at = torch.arange(seq, device="cuda")
        drop = torch.randint(0, max(1, seq // 3), (batch, 1), generator=gen, device="cuda")
        drop[0] = 0
        mask = ((at >= drop) if left else (at < seq - drop)).float()
    return mask


def _build(case, family):
    h, heads, depth = case["hidden"], case["heads"], case["depth"]
    env.load(mode=None)
    with torch.device("cuda"):
        if family == "gpt2":
            m = gpt2.GPT2(vocab_size=case["vocab"], max_position_embeddings=1024, hidden_size=h, num_heads=heads,
                          intermediate_size=4 * h, depth=depth, dropout=0.0, embedding_dropout=0.0, init_std=0.02,
                          checkpoint=case.get("ckpt", False))
        elif family == "vit":
            m = vit.VisionTransformer(img_size=case["img"], patch_size=case["patch"], num_classes=case["classes"], depth=depth,
                                      hidden_size=h, num_heads=heads, intermediate_size=4 * h, dropout=0.0)
        else:
            m = opt.OPT(vocab_size=case.get("vocab", VOCAB), hidden_size=h, num_hidden_layers=depth, ffn_dim=4 * h,
                        num_attention_heads=heads, max_position_embeddings=2048, dropout=0.0, init_std=0.02,
                        gradient_checkpointing=case.get("ckpt", False),
                        dtype=torch.bfloat16 if case.get("params") == "16bit" else None)
    return _settle(m)


def _batch(case, family, gen):
    if family == "vit":
        return dict(pixel_values=torch.randn(case["batch"], 3, case["img"], case["img"], generator=gen, device="cuda"),
                    labels=torch.randint(0, case["classes"], (case["batch"], ), generator=gen, device="cuda"))
    ids = torch.randint(2, case["vocab"], (case["batch"], case["seq"]), generator=gen, device="cuda")
    mask = _mask(case, gen)
    labels = ids.masked_fill(mask == 0, -100) if case["pad"] else ids.clone()
    return dict(input_ids=ids, attention_mask=mask, labels=labels)


def _loss_of(family):
    return {"gpt2": gpt2.GPT2LMLoss, "opt": opt.OPTLMLoss, "vit": cube_nn.CrossEntropyLoss}[family]()


def _vit_forward(model, batch):
    return model(batch["pixel_values"]), batch["labels"]


def _opt_forward(model, batch):
    return model(batch["input_ids"], batch["attention_mask"])[0], batch["labels"]


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        env.load(mode=None)
        dt = DTYPES[case["dtype"]]
        with torch.device("cuda"):
            layer = cube_nn.Linear(case["fan_in"], case["fan_out"], activation=case["act"] or None,
                                   weight_initializer=cube_nn.init.normal_(std=1 / math.sqrt(case["fan_in"])),
                                   bias_initializer=cube_nn.init.normal_(std=0.1))
        x = torch.randn(case["rows"], case["fan_in"], generator=gen, device="cuda").to(dt).requires_grad_(True)
        dy = torch.randn(case["rows"], case["fan_out"], generator=gen, device="cuda").to(dt)
        return dict(kind=kind, layer=layer, x=x, dy=dy, dtype=dt)
    family = _family(case)
    model = _build(case, family)
    if kind in ("prefill", "decode"):
        model.eval()
        cast = (lambda: torch.autocast("cuda", dtype=torch.bfloat16)) if case["params"] == "master" else contextlib.nullcontext
        ids = torch.randint(2, VOCAB, (case["batch"], case["seq"]), generator=gen, device="cuda")
        mask = _mask(case, gen, left=True) if case["pad"] else None
        state = dict(kind=kind, model=model, cast=cast, ids=ids, mask=mask, past=None)
        if kind == "decode":
            # the cache as the framework leaves it after the prompt and one further token
            _next_token(state, case["batch"], gen)
            _next_token(state, case["batch"], gen)
        return state
    batch, crit = _batch(case, family, gen), _loss_of(family)
    # a GPT-2 recipe's learning rate, weight decay and clipping; the scaler is only made for fp16
    trainer = Trainer(model, crit, FusedAdamW(model.parameters(), lr=3e-4, weight_decay=0.01), amp_dtype=DTYPES[case["dtype"]],
                      clip=None if kind == "vit" else 1.0, scaler_kwargs=dict(init_scale=2.0**12),
                      forward_fn={"gpt2": None, "vit": _vit_forward, "opt": _opt_forward}[family])
    params = list(model.parameters())
    return dict(kind=kind, trainer=trainer, batch=batch, params=params, moments=kind == "gpt2" and len(params) <= 30)


def _next_token(s, batch, gen):
    """Run the pass that ``s`` describes; ``s`` is then the pass of the token that follows."""
    s["past"] = _cached(s)[1]
    s["ids"] = torch.randint(2, VOCAB, (batch, 1), generator=gen, device="cuda")
    if s["mask"] is not None:
        s["mask"] = torch.cat([s["mask"], s["mask"].new_ones(batch, 1)], 1)


# ------------------------------------------------------------------------------------------------------ one pass
def _cached(s):
    with torch.no_grad(), s["cast"]():
        return s["model"](s["ids"], s["mask"], past_key_values=s["past"], use_cache=True)


def run(s):
    kind = s["kind"]
    if kind == "linear":
        layer, x = s["layer"], s["x"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        with torch.autocast("cuda", dtype=s["dtype"]):
            y = layer(x)
        y.backward(s["dy"])
        return y, x.grad, layer.weight.grad, layer.bias.grad
    if kind in ("prefill", "decode"):
        return _cached(s)
    if kind == "eval":
        logits, _, loss = s["trainer"].evaluate(s["batch"])
        return logits, loss
    loss, params = s["trainer"].step(s["batch"]), s["params"]
    out = dict(loss=loss, weights=[p.detach() for p in params])
    if s["moments"]:
        out["first_moments"] = [s["trainer"].optimizer.state[p]["exp_avg"] for p in params]
    return out


# ------------------------------------------------------------------------------------------------------ work
def work(case):
    """Bytes of the inputs and outputs once each, and the matrix products' operations (a causal mask halves attention; a
    recomputed block counts once)."""
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["rows"], case["fan_in"], case["fan_out"]
        return dict(bytes=2.0 * (2 * m * k + 2 * m * n) + 8.0 * (k * n + n), flops=6.0 * m * k * n)
    family = _family(case)
    h, depth, batch = case["hidden"], case["depth"], case["batch"]
    layers = depth * (12.0 * h * h + 13 * h)
    if family == "vit":
        n = (case["img"] // case["patch"])**2
        t, tokens = n + 1, batch * (n + 1)
        patch, head = 3.0 * case["patch"]**2 * h, float(case["classes"] * h)
        params = layers + patch + head + t * h
        flops = 2.0 * tokens * depth * 12 * h * h + 4.0 * batch * t * t * h * depth + 2.0 * batch * n * patch + 2.0 * batch * head
        inputs, logits = 12.0 * batch * case["img"]**2, 2.0 * batch * case["classes"]
    else:
        vocab = case.get("vocab", VOCAB)
        t = 1 if kind == "decode" else case["seq"]
        tokens = batch * t
        keys = case["seq"] + 2 if kind == "decode" else t / 2
        params = layers + (vocab + (1024 if family == "gpt2" else 2050)) * h
        flops = 2.0 * tokens * (depth * 12 * h * h + vocab * h) + 4.0 * tokens * keys * h * depth
        inputs, logits = 8.0 * tokens, 2.0 * tokens * vocab
    if kind in ("gpt2", "vit", "opt"):    # weights and both moments in and out
        return dict(bytes=24.0 * params + inputs, flops=3.0 * flops)
    cache = 0.0
    if kind == "prefill":
        cache = 4.0 * tokens * h * depth
    elif kind == "decode":                # the cache comes in and goes out one token longer
        cache = 8.0 * batch * (case["seq"] + 1.5) * h * depth
        params -= 2050.0 * h              # a few rows of the position table; the tied token table is read by the head
    return dict(bytes=2.0 * params + cache + logits + inputs, flops=flops)


def tolerance(case):
    """About four times the distance to the same pass through PyTorch's own kernels (other summation orders and roundings at
    the same precision), as measured over these cases and a dozen drawn ones."""
    if case["kind"] == "linear":          # 2.7e-3 to 3.4e-3: one rounding to 16 bits
        return {"rel": 0.013, "max": 0.06}
    if case["kind"] in ("gpt2", "vit", "opt"):   # weights up to 7.2e-3, first moments 6.8e-3
        return {"rel": 0.025, "max": 0.5}
    return {"rel": 0.03, "max": 0.4}      # logits and caches behind 12 to 24 layers in 16 bits: up to 1.6e-2

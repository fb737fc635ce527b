"""The work that users have this framework do, as cases that can be timed and compared.

Kinds: ``train`` and ``moe`` are one optimizer step of ``Trainer.train_step`` (forward, backward, clip, AdamW); ``prefill`` is
``TPDecoder.prefill`` of an OIL4 decoder over a paged cache; ``generate`` is ``TPDecoder.generate``, prompt in, tokens out; ``decode`` and
``prompts`` are ``Generator.step`` of a layer-list decoder (one token per sequence, and prompts of unequal length in one packed step);
``quantise`` is ``quantize_weight`` and back. Sizes are those of the presets, of ``bench.py`` and its companions and of the tests; deep models
keep their widths and are cut to a few layers, every layer being the same work; vocabularies of the OIL4 decoders are the byte one and the
64 M decoder's."""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from innova_b200.inference.generator import Generator
from innova_b200.models import PRESETS, DenseModel, MoEModel
from innova_b200.models.mekazen import MekazenConfig, MekazenModel
from innova_b200.ops.oil_linear import quantize_weight
from innova_b200.parallel.tp import TPDecoder
from innova_b200.training.trainer import TrainConfig, Trainer

DEV = "cuda"
LR, DECAY, CLIP = 3e-4, 0.1, 1.0
MEKAZEN = {"1k": (1024, 2816, 8, 2, 32768), "2k": (2048, 5632, 16, 4, 32768)}      # width, MLP, heads, key heads (head size 128), vocabulary


def listed():
    return [
        # the tiny train-in-format decoder: a step of about two hundred short launches
        dict(name="train_tiny_oil8", kind="train", preset="tiny", layers=4, batch=8, seq=128, ste="oil8", ckpt=False),
        # the 64 M decoder at an odd batch and an odd length, as a ragged text loader gives
        dict(name="train_64m_ragged", kind="train", preset="dense-64m", layers=14, batch=3, seq=1001, ste="", ckpt=False),
        # wide gated layers trained in format with gradient checkpointing, the 13 B recipe at a width that fits a single GPU's test
        dict(name="train_wide_oil8_ckpt", kind="train", preset="moe-24l", layers=2, batch=2, seq=2048, ste="oil8", ckpt=True),
        # the headline: GPT-2-small shape, 64 x 1024 tokens
        dict(name="train_gpt2_small", kind="train", preset="gpt2-small", layers=12, batch=64, seq=1024, ste="", ckpt=False),
        # a layer of the 24-layer mixture of experts, two sequences
        dict(name="train_moe", kind="moe", layers=1, batch=2, seq=2048, experts=8),
        # a short question to the 7 B decoder's layers: the time to the first token
        dict(name="prefill_1x77", kind="prefill", width=4096, layers=4, batch=1, prompt=77, cache="oil4"),
        # the headline's prompts
        dict(name="prefill_64x512", kind="prefill", width=4096, layers=4, batch=64, prompt=512, cache="oil4"),
        # a single user's answer; 16-bit cache
        dict(name="generate_1x32_64", kind="generate", width=2048, layers=8, batch=1, prompt=32, new=64, cache="bf16"),
        # many users' answers at the headline's batch and prompt
        dict(name="generate_64x512_64", kind="generate", width=2048, layers=8, batch=64, prompt=512, new=64, cache="oil4"),
        # one step of a running batch over contexts of unequal length
        dict(name="decode_mekazen_16", kind="decode", size="2k", layers=8, batch=16, context=1500, chunk=4096),
        # waiting requests admitted in one packed step
        dict(name="prompts_mekazen_5", kind="prompts", size="2k", layers=8, batch=5, tokens=3001, chunk=1024),
        # quantising one FFN matrix of the 7 B decoder and expanding it again
        dict(name="quantise_11008x4096", kind="quantise", rows=11008, cols=4096, fmt="oil4", dtype="float32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "moe", "prefill", "prefill", "generate", "generate", "decode", "prompts", "quantise"])
    if kind == "train":
        preset = rng.choice(["tiny", "dense-64m", "gpt2-small", "moe-24l"])
        layers = {"tiny": 4, "dense-64m": rng.randint(2, 14), "gpt2-small": rng.randint(2, 12), "moe-24l": rng.randint(1, 2)}[preset]
        most = {"tiny": 65536, "dense-64m": 32768, "gpt2-small": 32768, "moe-24l": 8192}[preset]
        seq = _log(rng, 17, PRESETS[preset]().max_seq_len)
        batch = max(1, _log(rng, 128, most) // seq)
        return dict(kind=kind, preset=preset, layers=layers, batch=batch, seq=seq, ste=rng.choice(["", "oil8", "oil4"]), ckpt=rng.random() < 0.25)
    if kind == "moe":
        seq = _log(rng, 33, 2048)
        return dict(kind=kind, layers=1, batch=max(1, _log(rng, 256, 8192) // seq), seq=seq, experts=rng.choice([4, 8]))
    if kind == "prefill":
        prompt = _log(rng, 5, 1100)
        return dict(kind=kind, width=rng.choice([2048, 4096]), layers=rng.randint(1, 4), batch=min(64, max(1, _log(rng, 8, 32768) // prompt)),
                    prompt=prompt, cache=rng.choice(["oil4", "bf16"]))
    if kind == "generate":
        return dict(kind=kind, width=2048, layers=rng.randint(1, 8), batch=_log(rng, 1, 64), prompt=_log(rng, 5, 512), new=_log(rng, 8, 128),
                    cache=rng.choice(["oil4", "bf16"]))
    if kind == "decode":
        return dict(kind=kind, size=rng.choice(["1k", "2k"]), layers=rng.randint(2, 8), batch=_log(rng, 1, 64), context=_log(rng, 40, 4000),
                    chunk=rng.choice([1024, 4096]))
    if kind == "prompts":
        batch = rng.randint(1, 9)
        return dict(kind=kind, size=rng.choice(["1k", "2k"]), layers=rng.randint(2, 8), batch=batch, tokens=_log(rng, 20 * batch, 8000),
                    chunk=rng.choice([1024, 4096]))
    return dict(kind=kind, rows=_log(rng, 64, 16000), cols=64 * _log(rng, 4, 160), fmt=rng.choice(["oil4", "oil8", "spark", "oil1"]),
                dtype=rng.choice(["float32", "bfloat16"]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, k=0):
    return torch.Generator(device=DEV).manual_seed(seed * 64 + k)


def _tokens(n, vocab, seed):
    """Zipf(1.1) token ids."""
    cdf = torch.arange(1, vocab + 1, dtype=torch.float64).pow(-1.1).cumsum(0)
    u = torch.rand(n, generator=_gen(seed, 1), device=DEV, dtype=torch.float64)
    return torch.searchsorted((cdf / cdf[-1]).to(DEV), u).clamp(max=vocab - 1)


def _lengths(total, n):
    """``n`` lengths of unequal size that add up to ``total``, each at least 1."""
    share = torch.rand(n, generator=torch.Generator().manual_seed(n)) + 0.25
    lens = [max(1, int(total * float(s))) for s in share / share.sum()]
    lens[-1] = max(1, total - sum(lens[:-1]))
    return lens


def _train_config(c):
    if c["kind"] == "moe":
        return PRESETS["moe-24l"](num_layers=c["layers"], num_experts=c["experts"], moe_ffn_hidden_size=5632)
    kw = dict(num_layers=c["layers"], ste_format=c["ste"], gradient_checkpointing=c["ckpt"])
    if c["preset"] == "moe-24l":          # its dense form: the same widths, one gated FFN per layer
        kw.update(num_experts=0)
    return PRESETS[c["preset"]](**kw)


def _prepare_train(c, seed):
    cfg = _train_config(c)
    model = (MoEModel if c["kind"] == "moe" else DenseModel)(cfg, dtype=torch.bfloat16, device=DEV, seed=seed)
    toks = _tokens(c["batch"] * c["seq"] + 1, cfg.vocab_size, seed)
    return dict(case=c, trainer=Trainer(model, TrainConfig(lr=LR, weight_decay=DECAY, max_grad_norm=CLIP)),
                ids=toks[:-1].view(c["batch"], c["seq"]).contiguous(), labels=toks[1:].view(c["batch"], c["seq"]).contiguous())


def _oil_config(c):
    if c["width"] == 4096:
        return PRESETS["llama-7b"](num_layers=c["layers"], vocab_size=256)
    return PRESETS["moe-24l"](num_layers=c["layers"], num_experts=0, num_kv_heads=4, vocab_size=8192)


def _prepare_oil(c, seed):
    cfg = _oil_config(c)
    dec = TPDecoder(cfg, fmt="oil4", max_batch=c["batch"], max_seq=c["prompt"] + c.get("new", 0) + 16, seed=seed, kv_format=c["cache"], single=True)
    # As in a trained model the next token is decided by clear margins: row t of the head points along the embedding of another
    # token, and embeddings outweigh what the few random layers add to them.
    dec.emb = (torch.randn(dec.emb.shape, generator=_gen(seed, 2), device=DEV) * 4.0).bfloat16()
    perm = torch.randperm(cfg.vocab_size, generator=_gen(seed, 3), device=DEV)
    dec.head = quantize_weight(dec.emb[perm].float() * (0.32 / cfg.hidden_size ** 0.5), "oil4")
    return dict(case=c, dec=dec, ids=_tokens(c["batch"] * c["prompt"], cfg.vocab_size, seed).view(c["batch"], c["prompt"]))


def _mekazen_dict(c):
    E, ff, H, G, V = MEKAZEN[c["size"]]
    rot = {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
    layer = {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": c["chunk"]},
                                            "rot": rot}, "mlp": {"kind": "dense", "ff": ff}}
    return {"vocab": V, "width": E, "layers": [layer] * c["layers"], "norm": {"eps": 1e-5}, "logit_softcap": 30.0, "max_seq_len": 8192 + 64}


def _mekazen_weights(d, seed):
    g, t = _gen(seed, 4), {}
    for n, shp in MekazenConfig.from_dict(d).tensor_shapes().items():
        x = torch.randn(shp, generator=g, device=DEV)
        if len(shp) == 1:
            x = x * 0.1 + (1.0 if n.endswith((".q.norm", ".k.norm")) else 0.0)
        elif n != "embed":
            x = x * shp[-1] ** -0.5
        t[n] = x.bfloat16().float() if len(shp) > 1 else x
    return t


def _prepare_mekazen(c, seed):
    d = _mekazen_dict(c)
    model = MekazenModel(MekazenConfig.from_dict(d), device=DEV)
    model.load_tensors(_mekazen_weights(d, seed))
    decode = c["kind"] == "decode"
    total = c["batch"] * c["context"] if decode else c["tokens"]
    lens = _lengths(total, c["batch"])
    if decode:
        lens = [min(n, 8192) for n in lens]
    pages = sum(n // 16 + 2 for n in lens) + 16
    gen = Generator(model, max_batch=c["batch"], max_seq=8192 + 64, num_pages=pages)
    flat = _tokens(sum(lens) + c["batch"], d["vocab"], seed).tolist()
    prompts, at = [], 0
    for n in lens:
        prompts.append(flat[at:at + n])
        at += n
    s = dict(case=c, gen=gen, prompts=prompts, rows=list(range(c["batch"])), zeros=[0] * c["batch"])
    if decode:
        for r, p in enumerate(prompts):
            gen.step([p], [0], [r], want=[])
        s.update(new=[[t] for t in flat[at:]], start=lens)
        for _ in range(3):                 # the batch has been running: its step is captured
            gen.step(s["new"], s["start"], s["rows"])
    return s


def prepare(case, seed):
    k = case["kind"]
    if k in ("train", "moe"):
        return _prepare_train(case, seed)
    if k in ("prefill", "generate"):
        return _prepare_oil(case, seed)
    if k in ("decode", "prompts"):
        return _prepare_mekazen(case, seed)
    w = torch.randn(case["rows"], case["cols"], generator=_gen(seed), device=DEV) * 0.02
    return dict(case=case, w=w.to(getattr(torch, case["dtype"])))


# ------------------------------------------------------------------------------------------------ one pass
def _cache_out(cache):
    if cache.fmt == "oil4":
        return {"k": list(cache.k_scale), "v": list(cache.v_scale)}
    return {"k": [p.view(torch.bfloat16) for p in cache.k_pool], "v": [p.view(torch.bfloat16) for p in cache.v_pool]}


def run(state):
    c = state["case"]
    k = c["kind"]
    if k in ("train", "moe"):
        t = state["trainer"]
        loss = t.train_step(state["ids"], state["labels"])
        return {"loss": loss, "master": t.engine.master, "exp_avg": t.engine.exp_avg, "exp_avg_sq": t.engine.exp_avg_sq, "weights": t.engine.flat_param}
    if k == "prefill":
        dec = state["dec"]
        return {"logits": dec.prefill(state["ids"]), "cache": _cache_out(dec.cache)}
    if k == "generate":
        dec = state["dec"]
        return {"tokens": dec.generate(state["ids"], c["new"])[0], "cache": _cache_out(dec.cache)}
    if k == "decode":
        gen = state["gen"]
        return {"logits": gen.step(state["new"], state["start"], state["rows"]), "cache": list(gen.cache.kv)}
    if k == "prompts":
        gen = state["gen"]
        for r in state["rows"]:
            gen.cache.free(r)
        return {"logits": gen.step(state["prompts"], state["zeros"], state["rows"]), "cache": list(gen.cache.kv)}
    qw = quantize_weight(state["w"], c["fmt"])
    return {"codes": qw.idx, "scales": qw.scales, "values": qw.dequantize()}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_params(cfg):
    E, D = cfg.hidden_size, cfg.head_dim
    attn = E * (cfg.num_heads + 2 * cfg.kv_heads) * D + cfg.num_heads * D * E
    return attn, (3 if cfg.activation == "silu" else 2) * E * cfg.ffn_hidden_size


def work(case):
    c, k = case, case["kind"]
    if k in ("train", "moe"):
        cfg = _train_config(c)
        T = c["batch"] * c["seq"]
        attn, ffn = _layer_params(cfg)
        experts = cfg.num_experts if k == "moe" else 1
        used = cfg.num_layers * (attn + ffn * (min(cfg.top_k, experts) if k == "moe" else 1)) + cfg.vocab_size * cfg.hidden_size
        params = cfg.num_layers * (attn + ffn * experts) + 2 * cfg.vocab_size * cfg.hidden_size
        score = 2 * c["batch"] * c["seq"] ** 2 // 2 * 2 * cfg.num_heads * cfg.head_dim * cfg.num_layers      # causal QK^T and PV
        # master, both moments read and written, the 16-bit weights read by the pass and written by the optimizer
        return {"bytes": params * 28.0 + 16.0 * T, "flops": 6.0 * used * T + 3.0 * score}
    if k in ("prefill", "generate"):
        cfg = _oil_config(c)
        attn, ffn = _layer_params(cfg)
        B, S, new = c["batch"], c["prompt"], c.get("new", 1)
        mats, head = cfg.num_layers * (attn + ffn), cfg.vocab_size * cfg.hidden_size
        wb = (mats + head) * 0.5625
        tok = 2 * cfg.num_layers * cfg.kv_heads * cfg.head_dim * (0.5625 if c["cache"] == "oil4" else 2.0)
        seen = sum(S + i for i in range(1, new))
        score = 4 * cfg.num_heads * cfg.head_dim * cfg.num_layers
        return {"bytes": wb * new + tok * B * (S + seen + new) + B * cfg.vocab_size * 4.0,
                "flops": 2.0 * mats * B * (S + new - 1) + 2.0 * head * B * new + score * B * (S * S / 2 + seen)}
    if k in ("decode", "prompts"):
        E, ff, H, G, V = MEKAZEN[c["size"]]
        mats, head = c["layers"] * (E * (3 * H + G) * 128 + 3 * E * ff), V * E
        T = c["batch"] if k == "decode" else c["tokens"]
        seen = c["batch"] * min(c["context"], c["chunk"]) if k == "decode" else T
        pairs = seen if k == "decode" else T * min(c["chunk"], T / c["batch"]) / 2
        return {"bytes": 2.0 * (mats + head) + 512.0 * G * c["layers"] * (seen + T) + 4.0 * c["batch"] * V,
                "flops": 2.0 * mats * T + 2.0 * head * c["batch"] + 4.0 * H * 128 * c["layers"] * pairs}
    n = c["rows"] * c["cols"]
    code = {"oil4": 0.5, "oil8": 1.0}.get(c["fmt"], 0.25)
    return {"bytes": n * ((4 if c["dtype"] == "float32" else 2) + 2 * (code + 0.0625) + 2), "flops": 0.0}


def tolerance(case):
    k = case["kind"]
    if k in ("train", "moe"):
        return {"rel": 0.02, "max": 0.9}
    if k == "quantise":
        return {"rel": 1e-5, "max": 1e-2, "differ": 1e-5}
    return {"rel": 0.02, "max": 0.5, "differ": 0.005}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _norm(x, w, b, cfg):
    return F.layer_norm(x, (x.shape[-1],), w, b, cfg.norm_eps) if cfg.norm == "layernorm" else _rms(x, w, cfg.norm_eps)


def _turn(x, first, theta):
    """Rotary positions, the two halves of a head as pairs; x [B, S, heads, D]."""
    half = x.shape[-1] // 2
    inv = theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    a = (first + torch.arange(x.shape[1], device=x.device, dtype=torch.float64)).view(1, -1, 1, 1) * inv
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _attend(q, k, v, scale, see):
    """q [B, S, H, D], k and v [B, N, G, D]; ``see`` [S, N] or [B, S, N] -> [B, S, H * D]."""
    B, S, H, D = q.shape
    G = k.shape[2]
    s = torch.einsum("bsgrd,bngd->bgrsn", q.view(B, S, G, H // G, D), k) * scale
    see = see if see.dim() == 2 else see[:, None, None]
    p = torch.softmax(s.masked_fill(~see, -math.inf), -1)
    return torch.einsum("bgrsn,bngd->bsgrd", p, v).reshape(B, S, H * D)


def _levels(fmt):
    if fmt == "oil8":
        return torch.linspace(-1.0, 1.0, 256, device=DEV).double()
    x = [0.1260, 0.3976, 0.6508, 0.9275, 1.2392, 1.5995, 2.0522, 2.7178]
    return (torch.tensor([-v for v in reversed(x)] + x, device=DEV) / 2.7178).double()


def _blocks(w, fmt):
    """(values, scales) of the block-32 formats in 64 bits."""
    b = w.double().reshape(-1, 32)
    mag = b.abs()
    top = mag.amax(-1, keepdim=True)
    if fmt in ("oil8", "oil4"):
        cb = _levels(fmt)
        i = torch.bucketize(b / top.clamp(min=1e-10), (cb[1:] + cb[:-1]) / 2)
        return (cb[i] * top).view(w.shape), top
    if fmt == "spark":
        keep = mag > 0.5 * top
        s = (mag * keep).sum(-1, keepdim=True) / keep.sum(-1, keepdim=True).clamp(min=1)
        return (b.sign() * keep * s).view(w.shape), s
    s = mag.mean(-1, keepdim=True)
    return torch.where(b >= 0, s, -s).view(w.shape), s


def _exact_train(c, seed):
    s = _prepare_train(c, seed)
    eng, cfg = s["trainer"].engine, _train_config(c)
    total = eng.total
    start = {n: p.detach().double() for n, p, _, _ in eng.entries}
    grads = {n: torch.zeros_like(w) for n, w in start.items()}
    places = [(n, o, k) for n, _, o, k in eng.entries]
    decay_end, ids, labels = eng.decay_end, s["ids"], s["labels"]
    del s, eng
    ste = c.get("ste", "")
    H, G, D, E = cfg.num_heads, cfg.kv_heads, cfg.head_dim, cfg.hidden_size
    w = {n: (_blocks(t, ste)[0] if ste and t.dim() == 2 and "embeddings" not in n else t).requires_grad_() for n, t in start.items()}

    def lin(x, name, bias=True):
        return F.linear(x, w[name + ".weight"], w.get(name + ".bias") if bias else None)

    T = ids.numel()
    see = torch.ones(c["seq"], c["seq"], dtype=torch.bool, device=DEV).tril()
    at_once = ids.shape[0] if c["kind"] == "moe" else max(1, min(ids.shape[0], 4096 // c["seq"]))
    loss_sum = torch.zeros((), dtype=torch.float64, device=DEV)
    for b0 in range(0, ids.shape[0], at_once):
        tok, lab = ids[b0:b0 + at_once], labels[b0:b0 + at_once]
        B, S = tok.shape
        x = w["tok_embeddings.weight"][tok]
        if "pos_embeddings.weight" in w:
            x = x + w["pos_embeddings.weight"][:S]
        aux = 0.0
        for i in range(cfg.num_layers):
            p = f"layers.{i}."
            qkv = lin(_norm(x, w[p + "attention_norm.weight"], w.get(p + "attention_norm.bias"), cfg), p + "attention.qkv_proj").view(B, S, -1, D)
            q, k, v = qkv.split([H, G, G], 2)
            if cfg.positions == "rope":
                q, k = _turn(q, 0, cfg.rope_theta), _turn(k, 0, cfg.rope_theta)
            x = x + lin(_attend(q, k, v, D ** -0.5, see), p + "attention.o_proj")
            h = _norm(x, w[p + "ffn_norm.weight"], w.get(p + "ffn_norm.bias"), cfg)
            if c["kind"] == "moe":
                h2 = h.reshape(-1, E)
                z = h2 @ w[p + "moe.router.weight"].t()
                prob = torch.softmax(z, -1)
                wt, idx = prob.topk(cfg.top_k, -1)
                y, share = torch.zeros_like(h2), []
                for e in range(cfg.num_experts):
                    row, col = (idx == e).nonzero(as_tuple=True)
                    share.append(row.numel() / idx.numel())
                    g, u = (h2[row] @ w[p + "moe.w_gate_up"][e].t()).chunk(2, -1)
                    y = y.index_add(0, row, (F.silu(g) * u) @ w[p + "moe.w_down"][e].t() * wt[row, col].unsqueeze(-1))
                aux = aux + cfg.lb_coef * cfg.num_experts * (prob.mean(0) * torch.tensor(share, device=DEV)).sum()
                aux = aux + cfg.z_coef * torch.logsumexp(z, -1).square().mean()
                x = x + y.view(x.shape)
            elif cfg.activation == "silu":
                g, u = lin(h, p + "ffn.gate_up_proj").chunk(2, -1)
                x = x + lin(F.silu(g) * u, p + "ffn.down_proj")
            else:
                x = x + lin(F.gelu(lin(h, p + "ffn.up_proj"), approximate="tanh"), p + "ffn.down_proj")
        h = _norm(x, w["norm.weight"], w.get("norm.bias"), cfg)
        z = F.linear(h, w["lm_head.weight"][: cfg.vocab_size]).reshape(-1, cfg.vocab_size)
        loss = F.cross_entropy(z, lab.reshape(-1), reduction="sum") / T + aux
        for n, g in zip(w, torch.autograd.grad(loss, list(w.values()))):
            grads[n] += g
        loss_sum += loss.detach()
        del x, h, z, loss
    norm = math.sqrt(sum(float(g.square().sum()) for g in grads.values()))
    clip = min(1.0, CLIP / (norm + 1e-6))
    out = {n: torch.zeros(total, dtype=torch.float64, device=DEV) for n in ("master", "exp_avg", "exp_avg_sq")}
    for n, o, k in places:
        g, p = grads.pop(n).reshape(-1) * clip, start[n].detach().reshape(-1)
        out["exp_avg"][o:o + k], out["exp_avg_sq"][o:o + k] = 0.1 * g, 0.001 * g.square()
        out["master"][o:o + k] = p * (1 - LR * (DECAY if o < decay_end else 0.0)) - LR * g / (g.abs() + 1e-8)
    return {"loss": loss_sum, **out, "weights": out["master"]}


def _exact_oil(c, seed):
    s = _prepare_oil(c, seed)
    dec, ids = s["dec"], s["ids"]
    cfg = dec.cfg
    H, G, D = cfg.num_heads, cfg.kv_heads, cfg.head_dim
    B, S = ids.shape

    def wide(qw):
        code = torch.stack([qw.idx & 15, qw.idx >> 4], -1).view(qw.N, -1).long()
        return (_levels("oil4")[code].view(qw.N, -1, 32) * qw.scales.double().unsqueeze(-1)).view(qw.N, -1)

    layers = [{n: wide(l[n]) for n in ("qkv", "o", "gu", "down")} for l in dec.layers]
    head, emb = wide(dec.head), dec.emb.double()
    kv = [[] for _ in layers]
    N = S + c.get("new", 1) - 1

    def forward(tok, first):
        x = emb[tok]
        n = tok.shape[1]
        see = torch.arange(first + n, device=DEV).view(1, -1) <= first + torch.arange(n, device=DEV).view(-1, 1)
        for l, seen in zip(layers, kv):
            q, k, v = (_rms(x, 1.0, cfg.norm_eps) @ l["qkv"].t()).view(tok.shape[0], n, -1, D).split([H, G, G], 2)
            q, k = _turn(q, first, cfg.rope_theta), _turn(k, first, cfg.rope_theta)
            seen.append((k, v))
            if c["cache"] == "oil4" and first:       # a decode step reads the cache as it is stored
                k, v = (torch.cat([_blocks(t[j].contiguous(), "oil4")[0] for t in seen], 1) for j in (0, 1))
            else:
                k, v = (torch.cat([t[j] for t in seen], 1) for j in (0, 1))
            a = torch.cat([_attend(q[i:i + 8], k[i:i + 8], v[i:i + 8], D ** -0.5, see) for i in range(0, tok.shape[0], 8)])
            x = x + a @ l["o"].t()
            g, u = (_rms(x, 1.0, cfg.norm_eps) @ l["gu"].t()).chunk(2, -1)
            x = x + (F.silu(g) * u) @ l["down"].t()
        return (_rms(x[:, -1], 1.0, cfg.norm_eps) @ head.t())[:, : cfg.vocab_size]

    step = max(1, 4096 // S)
    parts = []
    for b in range(0, B, step):                      # the prompts, a few sequences at a time
        before = [list(t) for t in kv]
        for t in kv:
            t.clear()
        parts.append(forward(ids[b:b + step], 0))
        for t, old in zip(kv, before):
            t[:] = [tuple(torch.cat([old[0][j], t[0][j]]) for j in (0, 1))] if old else t
    logits = torch.cat(parts)
    if c["kind"] == "generate":
        tok = logits.argmax(-1, keepdim=True)
        for i in range(c["new"] - 1):
            tok = forward(tok, S + i).argmax(-1, keepdim=True)
    # page p of row b and slot t hold position 16 * (p - first page of b) + t; pages are handed out in order, row after row
    pages = -(-dec.max_seq // 16)
    out = {"k": [], "v": []}
    for seen in kv:
        for j, name in enumerate(("k", "v")):
            t = F.pad(torch.cat([u[j] for u in seen], 1), (0, 0, 0, 0, 0, pages * 16 - N)).view(B * pages, 16, G, D).transpose(1, 2)
            out[name].append(t.reshape(B * pages, G, 16, -1, 32).abs().amax(-1) if c["cache"] == "oil4" else t.contiguous())
    return {"logits" if c["kind"] == "prefill" else "tokens": logits if c["kind"] == "prefill" else None, "cache": out}


def _exact_mekazen(c, seed):
    d = _mekazen_dict(c)
    w = {n: t.double() for n, t in _mekazen_weights(d, seed).items()}
    s = _prepare_mekazen(c, seed)
    prompts = [p + n for p, n in zip(s["prompts"], s["new"])] if c["kind"] == "decode" else s["prompts"]
    del s
    eps, m = d["norm"]["eps"], d["layers"][0]["mixer"]
    H, G, D, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
    f = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, device=DEV, dtype=torch.float64) / rot["dims"])
    z = rot["scaling"]
    keep = ((z["original"] * f / (2 * math.pi) - z["low"]) / (z["high"] - z["low"])).clamp(0, 1)
    f = (1 - keep) * f / z["factor"] + keep * f
    out = []
    for p in prompts:
        n = len(p)
        pos = torch.arange(n, device=DEV)
        see = (pos.view(1, -1) <= pos.view(-1, 1)) & (pos.view(1, -1) // c["chunk"] == pos.view(-1, 1) // c["chunk"])
        a = (pos.double().view(-1, 1) * f).unsqueeze(1)

        def turn(x):
            u, v = x[..., 0:rot["dims"]:2], x[..., 1:rot["dims"]:2]
            return torch.cat([torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2), x[..., rot["dims"]:]], -1)

        x = w["embed"][torch.tensor(p, device=DEV)]
        for i in range(c["layers"]):
            l = f"l{i}."
            h = _rms(x, 1 + w[l + "norm1"], eps)
            q, k = h @ w[l + "mix.q"].t(), h @ w[l + "mix.k"].t()
            v = k.view(1, n, G, D)
            q = turn(_rms(q, w[l + "mix.q.norm"], eps).view(n, H, D)).unsqueeze(0)
            k = turn(_rms(k, w[l + "mix.k.norm"], eps).view(n, G, D)).unsqueeze(0)
            o = torch.cat([_attend(q[:, j:j + 512], k, v, m["scale"], see[j:j + 512]) for j in range(0, n, 512)], 1)[0]
            y = (o * torch.sigmoid(h @ w[l + "mix.g"].t())) @ w[l + "mix.o"].t()
            x = x + _rms(y, 1 + w[l + "norm1b"], eps)
            h = _rms(x, 1 + w[l + "norm2"], eps)
            y = (F.silu(h @ w[l + "mlp.gate"].t()) * (h @ w[l + "mlp.up"].t())) @ w[l + "mlp.down"].t()
            x = x + _rms(y, 1 + w[l + "norm2b"], eps)
        t = _rms(x[-1], 1 + w["final.norm"], eps) @ w["head"].t()
        out.append(d["logit_softcap"] * torch.tanh(t / d["logit_softcap"]))
    return {"logits": torch.stack(out), "cache": [None] * c["layers"]}


def exact(case, seed):
    k = case["kind"]
    if k in ("train", "moe"):
        return _exact_train(case, seed)
    if k in ("prefill", "generate"):
        return _exact_oil(case, seed)
    if k in ("decode", "prompts"):
        return _exact_mekazen(case, seed)
    s = prepare(case, seed)
    values, scales = _blocks(s["w"], case["fmt"])
    return {"codes": None, "scales": scales.view(case["rows"], -1), "values": values}

"""``TPDecoder`` on one GPU against an fp64 forward over its own packed weights: prompts on either side of the packed route, steps of a few
tokens and of more, captured and eager, one decoder through calls of changing sizes."""
import gc

import pytest
import torch

from innova_b200.models import TransformerConfig

pytestmark = pytest.mark.gpu


def decoder(kv, **kw):
    """A small decoder whose layers count: weights of the size that keeps a row's norm, biases, norm weights off one."""
    from innova_b200.ops.oil_linear import quantize_weight
    from innova_b200.parallel.tp import TPDecoder
    cfg = TransformerConfig(vocab_size=500, hidden_size=256, num_layers=3, num_heads=4, head_dim=64, ffn_hidden_size=704, num_kv_heads=2, max_seq_len=512)
    dec = TPDecoder(cfg, max_batch=20, max_seq=288, seed=1, kv_format=kv, single=True, **kw)
    g = torch.Generator(device="cuda").manual_seed(2)

    def rand(*s):
        return torch.randn(*s, device="cuda", generator=g)

    for l in dec.layers:
        for k in ("qkv", "o", "gu", "down"):
            q = l[k]
            l[k] = quantize_weight(rand(q.N, q.K) * q.K ** -0.5, "oil4", bias=rand(q.N) * 0.1)
        l["n1"], l["n2"] = ((rand(256) * 0.2 + 1).bfloat16() for _ in range(2))
    dec.norm_w = (rand(256) * 0.2 + 1).bfloat16()
    dec.emb, dec.head = rand(*dec.emb.shape).bfloat16(), quantize_weight(rand(dec.head.N, 256) / 16, "oil4")
    torch.cuda.synchronize()
    return dec


def reference(dec, ids):
    """fp64 logits [B, S, vocab] of whole sequences."""
    cfg = dec.cfg
    B, S = ids.shape
    H, G, D = dec.H, dec.Hkv, dec.D

    def lin(x, q):
        y = x @ q.dequantize().double().t()
        return y if q.bias is None else y + q.bias.double()

    def norm(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.norm_eps) * w.double()

    def turn(x):
        c, s = (t[:S].double().view(S, 1, D // 2) for t in dec.rope)
        a, b = x.chunk(2, -1)
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    x = dec.emb[ids].double()
    for l in dec.layers:
        q, k, v = lin(norm(x, l["n1"]), l["qkv"]).view(B, S, H + 2 * G, D).split([H, G, G], 2)
        q, k, v = turn(q).transpose(1, 2), turn(k).transpose(1, 2), v.transpose(1, 2)
        a = torch.nn.functional.scaled_dot_product_attention(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), is_causal=True)
        x = x + lin(a.transpose(1, 2).reshape(B, S, H * D), l["o"])
        g, u = lin(norm(x, l["n2"]), l["gu"]).chunk(2, -1)
        x = x + lin(torch.nn.functional.silu(g) * u, l["down"])
    return lin(norm(x, dec.norm_w), dec.head)[..., :cfg.vocab_size]


def tokens(B, S, seed):
    return torch.randint(0, 500, (B, S), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


# Activations are rounded to bf16 some thirty times on the way, 2^-9 at most each, at random signs: 1.1e-2. A packed cache adds its 4 bits:
# levels lie a tenth to a quarter of a block's maximum (two deviations) apart, so keys and values are off by 0.075 of their size and the
# attention by 0.1; attention makes up to three quarters of the last residual.
LOGITS = {"bf16": 2e-2, "oil4": 0.12}


@pytest.mark.parametrize("kv", ["bf16", "oil4"])
@pytest.mark.parametrize("B,S", [(1, 1), (1, 128), (1, 129), (16, 8), (16, 9), (17, 40), (3, 250)])
def test_prompt_and_step_logits(kv, B, S, monkeypatch):
    """The prompt's logits, and a step's on the few-token route and on the tile product at the same batch."""
    from innova_b200.parallel import tp
    dec = decoder(kv)
    ids, nxt = tokens(B, S, S), tokens(B, 1, 7 * B)
    want = reference(dec, torch.cat([ids, nxt], 1))[:, -2:]

    def off(y, ref):
        return float((y.double() - ref).norm() / ref.norm())

    dec._splits, dec._scratch = 2, torch.empty(B * dec.H * 2 * (dec.D + 2), device="cuda")
    got = []
    for few in (True, False):
        if not few:
            monkeypatch.setattr(tp, "skinny_takes", lambda qw, M: False)
        assert off(dec.prefill(ids), want[:, 0]) < LOGITS["bf16"]      # a prompt attends over its own unpacked keys
        got.append(dec._decode_step(nxt[:, 0]))
        assert off(got[-1], want[:, 1]) < LOGITS[kv]
        assert dec.cache.seq_lens[:B].tolist() == [S + 1] * B
    assert off(got[0], got[1].double()) < 2e-2


@pytest.mark.parametrize("kv", ["bf16", "oil4"])
def test_generation_through_changing_sizes(kv):
    """One decoder, calls of changing batch, prompt and context (one split and several): every token, replayed or eager, is the best one of
    the fp64 forward over what came before it, up to the error of the logits. Wrong tokens lie about three deviations below."""
    dec = decoder(kv)
    for i, (B, S, new) in enumerate([(1, 32, 9), (16, 8, 7), (17, 8, 6), (1, 130, 5), (2, 200, 9), (20, 40, 4), (1, 32, 9), (16, 8, 1)]):
        ids = tokens(B, S, 100 + i)
        for graph in (True, False, True):
            out, _, _ = dec.generate(ids, new, use_graph=graph)
            assert out.shape == (B, new) and dec.cache.seq_lens[:B].tolist() == [S + new - 1] * B
            z = reference(dec, torch.cat([ids, out], 1))[:, S - 1:-1]
            behind = z.amax(-1) - z.gather(-1, out.unsqueeze(-1)).squeeze(-1)
            assert float(behind.max()) < 4 * LOGITS[kv] * float(z.std())


def test_a_step_takes_tokens_from_the_host():
    dec = decoder("bf16")
    dec._splits, dec._scratch = 1, torch.empty(1, device="cuda")
    got = []
    for dev in ("cuda", "cpu"):
        dec.prefill(tokens(3, 7, 5))
        got.append(dec._decode_step(tokens(3, 1, 6)[:, 0].contiguous().to(dev)))
    assert float((got[0] - got[1]).norm() / got[0].norm()) < 2e-2


def test_a_step_counts_tokens_from_the_end_and_reports_others():
    """As PyTorch's lookup: a negative token is a row from the end of the table, one outside it an error, here of the status word."""
    from innova_b200.ops import runtime as rt
    dec = decoder("bf16")
    dec._splits, dec._scratch = 1, torch.empty(1, device="cuda")
    rows = dec.emb.shape[0]

    def step(*t):
        dec.prefill(tokens(2, 5, 3))
        return dec._decode_step(torch.tensor(t, device="cuda"))

    want = step(rows - 1, 7)
    got = step(-1, 7)
    rt.check_status()
    assert float((got - want).norm() / want.norm()) < 2e-2
    for bad in (rows, -rows - 1, 2 ** 40):
        step(3, bad)
        with pytest.raises(RuntimeError, match="bad_arg"):
            rt.check_status()
    rt.check_status()


def test_the_route_of_a_step_follows_its_weights():
    """Too many tokens are told from the head alone; a matrix or norm off its alignment takes the whole step to the tile product."""
    from innova_b200.parallel import tp
    dec, asked = decoder("bf16"), []
    takes = tp.skinny_takes
    with pytest.MonkeyPatch.context() as m:
        m.setattr(tp, "skinny_takes", lambda qw, M: asked.append(qw) or takes(qw, M))
        assert not dec._few(17) and asked == [dec.head] and dec._few(16)
    down = dec.layers[1]["down"]
    moved = torch.empty(down.idx.numel() + 16, dtype=torch.uint8, device="cuda")[16:].view_as(down.idx).copy_(down.idx)
    ids = tokens(2, 30, 3)
    down.idx = moved
    assert not dec._few(2)
    got, _, _ = dec.generate(ids, 6)
    z = reference(dec, torch.cat([ids, got], 1))[:, 29:-1]
    assert float((z.amax(-1) - z.gather(-1, got.unsqueeze(-1)).squeeze(-1)).max()) < 4 * LOGITS["bf16"] * float(z.std())


@pytest.mark.parametrize("change", ["route", "width"])
def test_no_accumulator_comes_from_a_capture(change, monkeypatch):
    """A decoder whose step changes its route or a width after a call of the same batch: what the products keep for the process is
    allocated before the capture, not in it."""
    from innova_b200.ops import oil_linear as ol
    from innova_b200.ops.oil_linear import quantize_weight
    from innova_b200.parallel import tp
    B, S = (2, 6) if change == "route" else (18, 10)       # prompts that do not allocate them either
    dec, ids, taken = decoder("bf16"), tokens(B, S, 1), []
    monkeypatch.setattr(ol, "_acc", {})

    def spy(x, qw, M, make=ol._acc_for):
        missing = (x.device.index, qw.N) not in ol._acc
        taken.append(missing and torch.cuda.is_current_stream_capturing())
        return make(x, qw, M)

    monkeypatch.setattr(ol, "_acc_for", spy)
    monkeypatch.setattr(tp, "_acc_for", spy)
    dec.generate(ids, 2)
    if change == "route":
        q = dec.layers[0]["down"]
        q.idx = torch.empty(q.idx.numel() + 16, dtype=torch.uint8, device="cuda")[16:].view_as(q.idx).copy_(q.idx)
    else:
        dec.layers[1]["gu"], dec.layers[1]["down"] = (quantize_weight(torch.randn(*s, device="cuda") / 16, "oil4") for s in ((1280, 256), (256, 640)))
    dec.generate(ids, 1)
    assert taken and not any(taken) and all(not a.any() for a in ol._acc.values())


def test_a_collection_in_the_middle_of_a_capture():
    dec = decoder("bf16")
    ids = tokens(1, 12, 5)          # few enough for sums in a fixed order all the way
    want, _, _ = dec.generate(ids, 8)
    step = dec._decode_step

    def collecting(tok):
        out = step(tok)
        if torch.cuda.is_current_stream_capturing():
            gc.collect()
        return out

    class Ring:
        pass

    ring, graph = Ring(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = torch.zeros(4, device="cuda") + 1
    ring.me, ring.held = ring, (graph, y, torch.cuda.Event(), torch.empty(1 << 20, device="cuda"), torch.empty(1 << 16, pin_memory=True))
    ring.held[2].record()
    torch.cuda.synchronize()
    del ring, graph, y
    dec._decode_step = collecting
    got, _, _ = dec.generate(ids, 8)
    assert torch.equal(got, want)

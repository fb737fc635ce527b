"""Generation with the paged KV cache (CPU arithmetic here, GPU kernels under the gpu mark) and .oil export."""
import pytest
import torch

from innova_b200.formats import export, oil
from innova_b200.inference.generator import Generator
from innova_b200.inference.kv_cache import KV_LEVELS, PagedKVCache
from innova_b200.inference.sampler import Sampler, SamplingParams
from innova_b200.models import DenseModel, TransformerConfig, tiny_dense


def _greedy_no_cache(model, ids, n):
    out = []
    cur = ids.clone()
    for _ in range(n):
        nxt = model(cur)[:, -1].argmax(-1)
        out.append(nxt)
        cur = torch.cat([cur, nxt.view(-1, 1)], 1)
    return torch.stack(out, 1)


@pytest.mark.parametrize("style", ["llama", "gpt2"])
def test_cached_generation_matches_full_recompute_cpu(style):
    torch.manual_seed(0)
    if style == "llama":
        cfg = TransformerConfig(vocab_size=97, hidden_size=64, num_layers=2, num_heads=4, head_dim=16, ffn_hidden_size=96, num_kv_heads=2,
                                max_seq_len=64, vocab_pad_to=1)
    else:
        cfg = TransformerConfig(vocab_size=97, hidden_size=64, num_layers=2, num_heads=4, head_dim=16, ffn_hidden_size=96, max_seq_len=64,
                                activation="gelu", norm="layernorm", positions="learned", bias=True, vocab_pad_to=1)
    model = DenseModel(cfg, dtype=torch.float32).eval()
    ids = torch.randint(0, 97, (2, 9))
    ref = _greedy_no_cache(model, ids, 6)
    gen = Generator(model, kv_format="bf16", max_batch=2, max_seq=64)
    out = gen.generate_tokens(ids, max_new_tokens=6)
    assert out == ref.tolist()
    assert gen.stats.new_tokens == 12 and gen.stats.prompt_tokens == 18


def test_oil4_kv_cache_is_close_to_exact_cpu():
    torch.manual_seed(1)
    c = PagedKVCache(1, 2, 64, max_batch=1, max_seq=64, device="cpu", fmt="oil4")
    k = torch.randn(1, 20, 128)
    v = torch.randn(1, 20, 128)
    c.reserve(0, 20)
    c.append(0, k, v, [0], [0])
    c.commit([0], [20])
    kk, vv = c.gather(0, 0)
    assert kk.shape == (20, 2, 64)
    rel = (kk.reshape(20, 128) - k[0]).norm() / k[0].norm()
    assert 0.02 < float(rel) < 0.2  # 4-bit: lossy but close
    assert c.bytes_per_token() == 2 * 2 * (32 + 4)
    c.truncate(0, 10)
    assert c.lengths()[0] == 10 and len(c._host_pages[0]) == 1


def test_sampler_rules_cpu():
    logits = torch.tensor([[1.0, 3.0, 2.0, -1.0]])
    assert int(Sampler(SamplingParams()).sample(logits)) == 1
    s = Sampler(SamplingParams(repetition_penalty=4.0))
    assert int(s.sample(logits.clone(), torch.tensor([[1]]))) == 2  # 3.0/4 < 2.0
    s = Sampler(SamplingParams(temperature=1.0, top_k=2, seed=0))
    draws = {int(s.sample(logits)) for _ in range(50)}
    assert draws <= {1, 2}
    s = Sampler(SamplingParams(temperature=1.0, top_p=0.5, seed=0))
    assert {int(s.sample(logits)) for _ in range(30)} == {1}


def test_export_and_reload_roundtrip(tmp_path):
    torch.manual_seed(2)
    cfg = tiny_dense(num_layers=1, hidden_size=64, num_heads=2, head_dim=32, ffn_hidden_size=128, max_seq_len=32, ste_format="")
    model = DenseModel(cfg, dtype=torch.float32).eval()
    p = str(tmp_path / "m.oil")
    export.save_model(model, p, fmt="OIL32")
    assert oil.read_idx(p + "idx")[0] == "tok_embeddings.weight"
    again = export.load_model(p)
    ids = torch.randint(0, 256, (1, 8))
    assert torch.allclose(again(ids), model(ids), atol=1e-6)
    q = str(tmp_path / "m8.oil")
    nbytes = export.save_model(model, q, fmt="OIL8")
    assert nbytes < 0.4 * sum(p_.numel() for p_ in model.parameters()) * 4
    m8 = export.load_model(q)
    r = oil.OILReader(q)
    assert set(r.tensor_formats("layers.0.attention.q_proj.weight")) == {oil.OIL8}
    assert set(r.tensor_formats("layers.0.attention_norm.weight")) == {oil.OIL32}
    assert (m8(ids) - model(ids)).abs().max() < 0.5


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,D,H,Hkv", [("bf16", 64, 4, 4), ("oil4", 128, 8, 2), ("oil4", 64, 4, 1), ("bf16", 128, 4, 2)])
def test_gpu_paged_decode_matches_cpu_path(fmt, D, H, Hkv):
    torch.manual_seed(3)
    dev = torch.device("cuda", 0)
    B, S0 = 3, 37
    gc = PagedKVCache(1, Hkv, D, B, 256, dev, fmt)
    cc = PagedKVCache(1, Hkv, D, B, 256, "cpu", fmt)
    k = torch.randn(B, S0, Hkv * D).bfloat16()
    v = torch.randn(B, S0, Hkv * D).bfloat16()
    for c, kk, vv in ((gc, k.to(dev), v.to(dev)), (cc, k, v)):
        for b in range(B):
            c.reserve(b, S0)
        c.append(0, kk, vv, list(range(B)), [0] * B)
        c.commit(list(range(B)), [S0, S0 - 5, S0 - 20])
    kg, _ = gc.gather(0, 1)
    kc, _ = cc.gather(0, 1)
    assert torch.allclose(kg.cpu(), kc, atol=2e-2)
    q = torch.randn(B, H * D).bfloat16()
    og = gc.decode_attention(0, q.to(dev), H, D ** -0.5)
    oc = cc.decode_attention(0, q.float(), H, D ** -0.5)
    assert float((og.float().cpu() - oc).norm() / oc.norm()) < 3e-2


@pytest.mark.gpu
def test_gpu_sampler_and_generation():
    dev = torch.device("cuda", 0)
    logits = torch.randn(5, 32000, device=dev) * 3
    assert torch.equal(Sampler(SamplingParams()).sample(logits), logits.argmax(-1))
    s = Sampler(SamplingParams(temperature=0.8, top_k=5, seed=1))
    top5 = logits.topk(5, -1).indices
    for _ in range(5):
        t = s.sample(logits)
        assert all(int(t[b]) in top5[b].tolist() for b in range(5))
    s = Sampler(SamplingParams(temperature=1.0, top_p=0.3, seed=2))
    probs = torch.softmax(logits.float(), -1)
    t = s.sample(logits)
    sp, si = probs.sort(-1, descending=True)
    for b in range(5):
        n_keep = int(((sp[b].cumsum(0) - sp[b]) < 0.3).sum())
        assert int(t[b]) in si[b, : n_keep + 1].tolist()
    cfg = TransformerConfig(vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, head_dim=64, ffn_hidden_size=512, num_kv_heads=2,
                            max_seq_len=256)
    model = DenseModel(cfg, dtype=torch.bfloat16, device=dev).eval()
    ids = torch.randint(0, 512, (2, 40), device=dev)
    out_b = Generator(model, kv_format="bf16", max_batch=2, max_seq=256).generate_tokens(ids, 8)
    ref = _greedy_no_cache(model, ids, 8).tolist()
    agree = sum(a == b for x, y in zip(out_b, ref) for a, b in zip(x, y))
    assert agree >= 12  # bf16 ties may flip a late token
    out_q = Generator(model, kv_format="oil4", max_batch=2, max_seq=256).generate_tokens(ids, 8)
    assert len(out_q[0]) == 8


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["oil4", "bf16"])
@pytest.mark.parametrize("B,S,Hkv,D,start", [(1, 1, 1, 32, 0), (3, 37, 2, 64, 5), (2, 131, 4, 128, 16), (2, 50, 3, 96, 30), (64, 70, 8, 128, 0)])
def test_gpu_kv_append_whole_rows_as_single_values(fmt, B, S, Hkv, D, start):
    """The append of 16-byte pieces against the one that takes a value per lane (rows off 16 bytes), byte for byte: zero blocks,
    values on and beside the halfway points, infinities and what is no number among them."""
    dev = torch.device("cuda", 0)
    g = torch.Generator(device="cuda").manual_seed(B + S)
    kv = torch.randn(B, S, 2 * Hkv * D, device=dev, generator=g).bfloat16()
    flat = kv.view(-1)
    flat[: D // 2] = 0.0
    grid = torch.linspace(-1.0, 1.0, flat[D:].numel(), device=dev).bfloat16()
    flat[D:][::3] = grid[::3]
    if S > 30:
        kv[0, 3, 1], kv[0, 4, 2], kv[0, 5, 3] = float("inf"), float("nan"), -float("inf")
        kv[0, 6, 4], kv[0, 7] = 3e38, 1e-39
    odd = torch.empty(B * S * (2 * Hkv * D + 1) + 1, dtype=torch.bfloat16, device=dev)[1:].view(B, S, 2 * Hkv * D + 1)
    odd[..., : 2 * Hkv * D] = kv
    caches = []
    for src in (kv, odd):
        c = PagedKVCache(1, Hkv, D, B, S + start + 16, dev, fmt)
        c.reserve_rows(range(B), S + start)
        c.append(0, src[..., : Hkv * D], src[..., Hkv * D:2 * Hkv * D], list(range(B)), [start] * B)
        caches.append(c)
    for name in ("k_pool", "v_pool") + (("k_scale", "v_scale") if fmt == "oil4" else ()):
        a, b = (getattr(c, name)[0].view(torch.uint8) for c in caches)
        assert torch.equal(a, b), name


def test_kv_thresholds_are_the_first_floats_nearer_to_the_next_level():
    """The constants of the append kernels, in 32-bit arithmetic: each takes its level and the float below it does not."""
    import pathlib
    import re
    import numpy as np
    import innova_b200
    text = (pathlib.Path(innova_b200.__file__).parent / "csrc" / "paged_attn.cu").read_text()

    def table(name, parse):
        return np.array([parse(v.strip().rstrip("f")) for v in re.search(name + r"\[\d+\] = \{([^}]*)\}", text).group(1).split(",")], dtype=np.float32)

    levels, thr = table("c_kv_levels", float), table("KV_THRESHOLDS", float.fromhex)
    assert len(levels) == 16 and len(thr) == 15 and np.allclose(levels, KV_LEVELS.numpy(), atol=1e-6)
    for j in range(15):
        for x, takes in ((thr[j], True), (np.nextafter(thr[j], np.float32(-2)), False)):
            assert bool((levels[j + 1] - x) < (x - levels[j])) == takes, (j, x)


@pytest.mark.gpu
def test_gpu_kv_codes_beside_the_halfway_points():
    """Codes of both append kernels against the level that the halfway points give in 64 bits: the bf16 values around each of them, in blocks
    whose maximum is 1, so that the division is exact."""
    dev = torch.device("cuda", 0)
    mids = (KV_LEVELS.double()[1:] + KV_LEVELS.double()[:-1]) / 2
    mids[7] = 0.0
    bits = mids[mids != 0].bfloat16().view(torch.int16)
    near = torch.cat([(bits + d).view(torch.bfloat16) for d in (-2, -1, 0, 1, 2)] + [torch.tensor([0.0, 2.0 ** -20, -2.0 ** -20]).bfloat16()])
    rows = torch.zeros(-(-near.numel() // 31), 32, dtype=torch.bfloat16)
    flat = torch.zeros(rows.shape[0] * 31, dtype=torch.bfloat16)
    flat[: near.numel()] = near
    rows[:, 0], rows[:, 1:] = 1.0, flat.view(-1, 31)
    want = (rows.double().unsqueeze(-1) > mids).sum(-1)
    S = rows.shape[0]
    for pad in (0, 1):                                            # rows on 16 bytes, and off them
        kv = torch.zeros(1, S, 64 + pad, dtype=torch.bfloat16, device=dev)
        kv[0, :, :32] = kv[0, :, 32:64] = rows.to(dev)
        c = PagedKVCache(1, 1, 32, 1, S + 16, dev, "oil4")
        c.reserve(0, S)
        c.append(0, kv[..., :32], kv[..., 32:64], [0], [0])
        for pool, scale in ((c.k_pool, c.k_scale), (c.v_pool, c.v_scale)):
            raw = pool[0][c._host_pages[0]].reshape(-1, 16)[:S].cpu()
            assert torch.equal(torch.stack([raw & 15, raw >> 4], -1).view(S, 32).long(), want)
            assert bool((scale[0][c._host_pages[0]].reshape(-1)[:S] == 1).all())


def test_reserve_and_free_rows_as_one_by_one():
    for rows, lens in (([0, 1, 2], [33, 33]), ([2, 0], [5, 40]), ([1], [17, 64])):
        one, many = (PagedKVCache(1, 1, 32, 4, 64, "cpu", "bf16", num_pages=10) for _ in range(2))
        for n in lens:
            for b in rows:
                one.reserve(b, n)
            many.reserve_rows(rows, n)
        assert torch.equal(one.page_table, many.page_table) and one._free == many._free and one._host_pages == many._host_pages
        one.seq_lens.fill_(9), many.seq_lens.fill_(9)
        for b in rows:
            one.free(b)
        many.free_rows(rows)
        assert torch.equal(one.seq_lens, many.seq_lens) and one._free == many._free
    full = PagedKVCache(1, 1, 32, 4, 64, "cpu", "bf16", num_pages=5)
    with pytest.raises(MemoryError):
        full.reserve_rows([0, 1, 2], 40)
    assert len(full._host_pages[0]) == 3 and full.page_table[0, :3].tolist() == full._host_pages[0]


@pytest.mark.gpu
@pytest.mark.parametrize("D,H,Hkv,n,splits", [(128, 16, 4, 1, 1), (128, 16, 4, 97, 1), (64, 8, 1, 203, 1), (128, 16, 4, 203, 3), (64, 4, 4, 16, 1)])
def test_gpu_bf16_decode_attention_direct_and_split(D, H, Hkv, n, splits):
    """Against fp64 attention; the slots behind the last token hold what is no number and must not count. fp32 inside: what is left is
    the rounding of the result."""
    from innova_b200.ops import runtime as rt
    dev = torch.device("cuda", 0)
    g = torch.Generator(device="cuda").manual_seed(n)
    c = PagedKVCache(1, Hkv, D, 1, 256, dev, "bf16")
    for pool in (c.k_pool, c.v_pool):
        pool[0].view(torch.bfloat16).fill_(float("nan"))
    c.reserve(0, n)
    k, v = (torch.randn(1, n, Hkv * D, device=dev, generator=g).bfloat16() for _ in range(2))
    c.append(0, k, v, [0], [0])
    c.commit([0], [n])
    q = torch.randn(1, H * D, device=dev, generator=g).bfloat16()
    out = torch.empty_like(q)
    scr = torch.empty(H * splits * (D + 2), device=dev)
    rt.check(rt.lib().inv_paged_decode(q.data_ptr(), q.stride(0), c.page_table.data_ptr(), c.max_pages, c.seq_lens.data_ptr(), 1, H, Hkv, D,
                                       c.k_pool[0].data_ptr(), c.v_pool[0].data_ptr(), 0, 0, 0, D ** -0.5, out.data_ptr(), out.stride(0),
                                       scr.data_ptr(), splits, rt.stream_ptr()), "inv_paged_decode")
    qd, kd, vd = q.double().view(Hkv, H // Hkv, D), k.double().view(n, Hkv, D), v.double().view(n, Hkv, D)
    p = torch.softmax(torch.einsum("hgd,thd->hgt", qd, kd) * D ** -0.5, -1)
    ref = torch.einsum("hgt,thd->hgd", p, vd).reshape(1, -1)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.0 ** -8

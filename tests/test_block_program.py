"""The block whose launches are issued by one native call against its layers one by one: same output to the bit, gradients up to the order
of fp32 sums; the cases that have to go layer by layer do."""
import pytest
import torch

from innova_b200.models import DenseModel, PRESETS
from innova_b200.models import dense

DEV = "cuda"
GELU = dict(activation="gelu", norm="layernorm", positions="learned", bias=True)


def _model(**kw):
    base = dict(num_layers=2, vocab_size=512, max_seq_len=512, hidden_size=256, num_heads=4, head_dim=64, ffn_hidden_size=448)
    base.update(kw)
    torch.manual_seed(3)
    m = DenseModel(PRESETS["tiny"](**base), dtype=torch.bfloat16, device=DEV)
    with torch.no_grad():
        for n, p in m.named_parameters():
            if n.endswith("bias") or "norm" in n:
                p.add_(torch.randn_like(p) * 0.1)
    return m


def _pass(m, ids, fused, monkeypatch, main=True):
    calls = []
    with monkeypatch.context() as mp:
        real = dense.ops.block_forward
        mp.setattr(dense.ops, "block_forward", (lambda *a: calls.append(0) or real(*a)) if fused else (lambda *a: None))
        for p in m.parameters():
            p.grad = None
            if main:
                p.main_grad = torch.full(p.shape, 0.5, dtype=torch.float32, device=DEV)
            elif hasattr(p, "main_grad"):
                del p.main_grad
        x = m.hidden_states(ids)
        loss = m(ids, ids)
        loss.backward()
    grads = {n: (p.main_grad - 0.5 if main else p.grad.float()) for n, p in m.named_parameters()}
    return x.detach(), float(loss), grads, len(calls)


@pytest.mark.gpu
@pytest.mark.parametrize("main", [True, False])
@pytest.mark.parametrize("B,S,kw", [
    (2, 128, {}), (3, 77, dict(num_kv_heads=2)), (1, 1, {}), (2, 200, GELU), (5, 33, dict(GELU, ste_format="oil8")),
    (2, 96, dict(ste_format="oil4", num_kv_heads=1)), (2, 130, dict(gradient_checkpointing=True)), (2, 65, dict(GELU, gradient_checkpointing=True, ste_format="spark")),
    (1, 129, dict(hidden_size=1280, num_heads=5, head_dim=128, ffn_hidden_size=200, bias=True, ste_format="oil1"))])
def test_block_in_one_call_matches_its_layers(B, S, kw, main, monkeypatch):
    m = _model(**kw)
    ids = torch.randint(0, 512, (B, S), device=DEV)
    x1, l1, g1, n1 = _pass(m, ids, True, monkeypatch, main)
    x0, l0, g0, _ = _pass(m, ids, False, monkeypatch, main)
    assert n1 >= 4 and torch.equal(x1, x0) and l1 == l0
    for n in g0:
        # the fp32 sums of attention's dQ and of the weight gradients arrive in another order; dQ is rounded to bf16 behind them
        assert float((g1[n] - g0[n]).norm()) <= 2.0 ** -7 * float(g0[n].norm()) + 1e-7, n
        # nothing behind the last layer's attention passes through dQ: the same sums in fp32, in another order, and up to four roundings of each
        # (2^-25 of the 0.5 that the buffers start from)
        if main and n.startswith(("layers.1.ffn", "layers.1.attention.o_proj")):
            assert float((g1[n] - g0[n]).norm()) <= 1e-5 * float(g0[n].norm()) + 2.0 ** -23 * g0[n].numel() ** 0.5, n


@pytest.mark.gpu
def test_block_follows_what_changes_between_and_within_passes(monkeypatch):
    m = _model(**GELU)
    ids = torch.randint(0, 512, (2, 64), device=DEV)
    seen = []
    real = dense.ops.block_forward

    def spy(*a):
        y = real(*a)
        seen.append(y is not None)
        return y

    monkeypatch.setattr(dense.ops, "block_forward", spy)

    def routes():
        seen.clear()
        m(ids, ids).backward()
        return list(seen)

    assert routes() == [True, True]
    m.layers[0].attention.qkv_proj.weight.requires_grad_(False)          # frozen: its gradient must not be computed
    m.layers[0].attention.qkv_proj.weight.main_grad = g = torch.zeros(768, 256, device=DEV)
    assert routes() == [False, True] and float(g.abs().max()) == 0.0
    m.layers[0].attention.qkv_proj.weight.requires_grad_(True)
    hits = []
    h = m.layers[1].ffn.register_forward_hook(lambda *a: hits.append(1))
    assert routes() == [True] and hits == [1]                             # a hook inside the block fires
    h.remove()
    h = m.layers[1].register_forward_hook(lambda *a: hits.append(2))
    assert routes() == [True, True] and hits == [1, 2]                    # one on the block itself does too
    h.remove()
    m.layers[0].ffn.adapter = lambda act: act[..., :256] * 0
    assert routes() == [False, True]
    m.layers[0].ffn.adapter = None
    # a gradient buffer that is taken away between the passes is not written to; the gradient goes through autograd
    w = m.layers[1].ffn.up_proj.weight
    w.main_grad, w.grad = torch.zeros_like(w, dtype=torch.float32), None
    loss = m(ids, ids)
    old = w.main_grad
    del w.main_grad
    loss.backward()
    assert float(old.abs().max()) == 0.0 and w.grad is not None and float(w.grad.abs().max()) > 0
    # tensors that pass through saved-tensor hooks, and no graph at all
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)):
        loss = m(ids, ids)
    loss.backward()
    with torch.no_grad():
        assert torch.equal(m.hidden_states(ids), m.hidden_states(ids))
    x = torch.randn(2, 64, 512, device=DEV).bfloat16()[..., ::2]          # not contiguous: layer by layer, as before
    assert real(m.layers[0], x, None, None) is None and m.layers[0](x, None).shape == x.shape


@pytest.mark.gpu
def test_block_asks_parts_that_were_set_up_on_their_own(monkeypatch):
    """Another format for one part of a block, and steps that were replaced in their class, count as they do layer by layer."""
    import copy
    m = _model(**GELU)
    x = torch.randn(2, 64, 256, device=DEV).bfloat16()
    plain = m.layers[0](x, None)
    own = copy.copy(m.cfg)
    own.ste_format = "spark"
    m.layers[0].ffn.cfg = own
    got = m.layers[0](x, None)
    with monkeypatch.context() as mp:
        mp.setattr(dense.ops, "block_forward", lambda *a: None)
        want = m.layers[0](x, None)
    assert torch.equal(got, want) and not torch.equal(got, plain)
    m.layers[0].ffn.cfg = m.cfg
    calls, real = [], dense.Attention.forward
    monkeypatch.setattr(dense.Attention, "forward", lambda self, *a: calls.append(1) or real(self, *a))
    assert torch.equal(m.layers[0](x, None), plain) and calls == [1]
    monkeypatch.undo()
    m = _model(norm="rmsnorm")
    rope = m.rope(x.device)
    want = m.layers[0](x, rope)
    m.layers[0].ffn_norm.bias = torch.nn.Parameter(torch.ones_like(m.layers[0].ffn_norm.weight))     # nothing that an RMS norm reads
    assert torch.equal(m.layers[0](x, rope), want)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, GELU, dict(ste_format="oil8", num_kv_heads=2), dict(GELU, ste_format="oil4"), dict(hidden_size=128, num_heads=4, ffn_hidden_size=64)])
def test_block_without_gradients(kw, monkeypatch):
    """No graph: the same output, and no more memory at once than layer by layer (and the bytes by which buffers are rounded up)."""
    m = _model(**kw)
    x = torch.randn(4, 500, m.cfg.hidden_size, device=DEV).bfloat16()
    rope = m.rope(x.device)
    want = m.layers[0](x, rope)

    def peak():
        torch.cuda.synchronize()
        base = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        with torch.no_grad():
            y = m.layers[0](x, rope)
        torch.cuda.synchronize()
        assert torch.equal(y, want) and not y.requires_grad
        return torch.cuda.max_memory_allocated() - base

    once = peak()
    monkeypatch.setattr(dense.ops, "block_forward", lambda *a: None)
    assert once <= peak() + 64 * 1024


def test_block_buffers_are_sized_by_their_layout():
    """The bytes that the native side asks for, stated once more by hand, at sizes off the 256 bytes that buffers start on."""
    from innova_b200.ops import block
    up = lambda *n: sum((x + 255) // 256 * 256 for x in n)
    for B, S, E, H, Hkv, D, F, gated, q in ((1, 1, 64, 1, 1, 64, 8, 0, 0), (3, 77, 200, 4, 2, 64, 136, 1, 1), (2, 129, 1280, 5, 1, 128, 200, 0, 1)):
        T, W, O, mid = B * S, (H + 2 * Hkv) * D, H * D, 2 * F if gated else F
        weights = up(*(2 * q * n for n in (W * E, E * O, mid * E, E * F)))
        stats = up(4 * T * H) + 4 * up(4 * T)
        args = (B, S, E, H, Hkv, D, F, gated, q)
        assert block._bytes(block.SAVED, *args) == weights + up(2 * T * E, 2 * T * W, 2 * T * O, 2 * T * E, 2 * T * E, 2 * T * mid, 2 * T * F) + stats
        once = up(0 if O <= E else 2 * T * max(E, O)) + max(up(2 * T * W), up(2 * T * E, 2 * T * F, 2 * T * mid))
        assert block._bytes(block.FORWARD, *args) == up(2 * q * max(W * E, E * O, mid * E, E * F)) + once + up(4 * T * H) + 2 * up(4 * T)
        mlp = up(2 * T * mid) + (up(2 * T * F) if gated else 0)
        attn = up(up(4 * B * H * S) + 4 * T * O)
        grid = max(1, min(148, (T + 7) // 8))
        assert block._bytes(block.SCRATCH, *args) == max(mlp, up(2 * T * W)) + up(2 * T * E, 2 * T * E, 2 * T * O, 4 * E, grid * 3 * E * 4) + attn
    with pytest.raises(ValueError):
        block._bytes(block.SAVED, 0, 1, 64, 1, 1, 64, 8, 0, 0)


def test_block_cuts_its_weight_gradients_as_the_layers_do():
    from innova_b200.ops import block, runtime as rt  # noqa: F401
    from innova_b200.ops.gemm import _split_k_for
    for M in (8, 128, 129, 256, 257, 768, 2048, 11264):
        for N in (8, 128, 136, 264, 2048, 5632):
            for K in (1, 64, 65, 1024, 3003, 65536):
                assert rt.lib().inv_block_split_k(M, N, K) == _split_k_for(M, N, K), (M, N, K)


def test_train_step_puts_parts_in_eval_mode_back():
    from innova_b200.training.trainer import Trainer
    m = DenseModel(PRESETS["tiny"](num_layers=1, vocab_size=64, max_seq_len=16, hidden_size=32, num_heads=1, head_dim=32, ffn_hidden_size=32), dtype=torch.float32)
    t = Trainer(m)
    m.layers[0].ffn.eval()
    ids = torch.randint(0, 64, (1, 8))
    t.train_step(ids, ids)
    assert all(k.training for k in m.modules())

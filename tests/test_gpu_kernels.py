"""Numerics of every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return float((a - b).norm() / (b.norm() + 1e-12))


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    from innova_b200.ops import runtime as rt
    rt.check_status()


# ------------------------------------------------------------------------------------------ GEMM
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 776, 200), (1000, 264, 1032), (77, 8, 72)])
def test_gemm_layouts(a_mn, b_mn, M, N, K):
    from innova_b200 import ops
    torch.manual_seed(0)
    dev = _dev()
    if a_mn and M % 8:
        M = (M + 7) // 8 * 8
    A = torch.randn(M, K, device=dev).bfloat16()
    B = torch.randn(N, K, device=dev).bfloat16()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    out = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    ref = A.float() @ B.float().t()
    assert out.shape == (M, N)
    assert _rel_err(out, ref) < 1e-2


def test_gemm_epilogues():
    from innova_b200 import ops
    torch.manual_seed(1)
    dev = _dev()
    M, N, K = 512, 768, 320
    A = (torch.randn(M, K, device=dev) * 0.5).bfloat16()
    B = (torch.randn(N, K, device=dev) * 0.1).bfloat16()
    bias = torch.randn(N, device=dev).bfloat16()
    aux = torch.randn(M, N, device=dev).bfloat16()
    ref = A.float() @ B.float().t()
    # bias
    out = ops.gemm(A, B, bias=bias)
    assert _rel_err(out, ref + bias.float()) < 1e-2
    # gelu with pre-activation output
    pre = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    out = ops.gemm(A, B, epilogue=ops.EPI_GELU, bias=bias, aux_out=pre)
    assert _rel_err(pre, ref + bias.float()) < 1e-2
    assert _rel_err(out, F.gelu(ref + bias.float(), approximate="tanh")) < 1e-2
    # dgelu
    x = aux.float().requires_grad_(True)
    F.gelu(x, approximate="tanh").sum().backward()
    out = ops.gemm(A, B, epilogue=ops.EPI_DGELU, aux_in=aux)
    assert _rel_err(out, ref * x.grad) < 2e-2
    # gelu with its derivative as the second output, and the multiply that consumes it in the backward pass
    dg = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    out = ops.gemm(A, B, epilogue=ops.EPI_GELU_DG, bias=bias, aux_out=dg)
    xb = (ref + bias.float()).requires_grad_(True)
    F.gelu(xb, approximate="tanh").sum().backward()
    assert _rel_err(out, F.gelu(xb.detach(), approximate="tanh")) < 1e-2
    assert _rel_err(dg, xb.grad) < 1e-2
    wide = (torch.randn(M, N, device=dev) * 40).bfloat16()              # far outside the range where tanh has saturated
    xw = wide.float().requires_grad_(True)
    F.gelu(xw, approximate="tanh").sum().backward()
    out = ops.gemm(A, B, epilogue=ops.EPI_DGELU, aux_in=wide)
    assert torch.isfinite(out.float()).all() and _rel_err(out, ref * xw.grad) < 2e-2
    out = ops.gemm(A, B, epilogue=ops.EPI_MUL, aux_in=aux)
    assert _rel_err(out, ref * aux.float()) < 1e-2
    # residual add (aliasing the output)
    res = aux.clone()
    ops.gemm(A, B, out=res, epilogue=ops.EPI_ADD, bias=bias, aux_in=res)
    assert _rel_err(res, ref + bias.float() + aux.float()) < 1e-2
    # fp32 output and split-K accumulation
    out32 = ops.gemm(A, B, out_dtype=torch.float32)
    assert _rel_err(out32, ref) < 1e-2
    acc = torch.ones(M, N, device=dev, dtype=torch.float32)
    ops.gemm(A, B, out=acc, epilogue=ops.EPI_ATOMIC, split_k=3)
    assert _rel_err(acc, ref + 1.0) < 1e-2


@pytest.mark.parametrize("M,N,K", [(20000, 776, 192), (2 * 74 * 256 + 300, 520, 128), (1000, 136, 64)])
def test_gemm_second_operand_epilogues_tails(M, N, K):
    """Residual-add and GELU-backward epilogues on the CTA-pair kernel: more tiles than CTA pairs (the operand boxes are
    fetched one ahead, across tiles), ragged last row and column tiles, a strided second operand, output aliasing it."""
    from innova_b200 import ops
    torch.manual_seed(5)
    dev = _dev()
    A = (torch.randn(M, K, device=dev) * 0.5).bfloat16()
    B = (torch.randn(N, K, device=dev) * 0.1).bfloat16()
    big = torch.randn(M, N + 24, device=dev).bfloat16()
    aux = big[:, 8:8 + N]                      # row pitch N + 24, 16-byte aligned start
    ref = A.float() @ B.float().t()
    out = ops.gemm(A, B, epilogue=ops.EPI_ADD, aux_in=aux)
    assert _rel_err(out, ref + aux.float()) < 1e-2
    x = aux.float().requires_grad_(True)
    F.gelu(x, approximate="tanh").sum().backward()
    out = ops.gemm(A, B, epilogue=ops.EPI_DGELU, aux_in=aux)
    assert _rel_err(out, ref * x.grad) < 2e-2
    res = aux.contiguous()
    want = ref + res.float()
    ops.gemm(A, B, out=res, epilogue=ops.EPI_ADD, aux_in=res)
    assert _rel_err(res, want) < 1e-2


@pytest.mark.parametrize("M,N,K", [(129, 136, 72), (300, 264, 200), (2 * 74 * 256 + 33, 392, 64)])
@pytest.mark.parametrize("a_mn,b_mn,epi", [(False, False, "NONE"), (False, False, "GELU"), (False, False, "ADD"), (False, False, "GELU_DG"),
                                           (False, False, "ATOMIC"), (False, True, "NONE"), (False, True, "MUL"), (True, True, "ATOMIC")])
def test_gemm_fixed_epilogues_stay_inside_their_view(a_mn, b_mn, epi, M, N, K):
    """The CTA-pair kernels whose epilogue is compiled in: boxes that reach past the last row and column, outputs that are views of a wider
    buffer (nothing around them is touched), bias, alpha, more tiles than pairs. bf16 results carry one rounding of 2^-9 (2^-8 with the
    packed fp16 GELU); fp32 sums K * 2^-24."""
    from innova_b200 import ops
    torch.manual_seed(7)
    dev = _dev()
    Ma = (M + 7) // 8 * 8 if a_mn else M
    A = (torch.randn(Ma, K, device=dev) * 0.5).bfloat16()
    B = (torch.randn(N, K, device=dev) * 0.2).bfloat16()
    bias = torch.randn(N, device=dev).bfloat16()
    f32 = epi == "ATOMIC"
    buf = torch.full((Ma + 3, N + 24), 3.0, device=dev, dtype=torch.float32 if f32 else torch.bfloat16)
    out = buf[:Ma, 8:8 + N]
    aux = torch.randn(Ma, N + 8, device=dev).bfloat16()[:, :N]
    kw = dict(aux_in=aux) if epi in ("ADD", "MUL") else dict(aux_out=aux) if epi in ("GELU", "GELU_DG") else {}
    aux_before = aux.float().clone()
    use_bias = epi in ("NONE", "GELU", "ADD", "GELU_DG")
    ops.gemm(A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B, out=out, a_mn=a_mn, b_mn=b_mn, epilogue=getattr(ops, "EPI_" + epi),
             bias=bias if use_bias else None, alpha=0.5, **kw)
    x = 0.5 * (A.double() @ B.double().t()) + (bias.double() if use_bias else 0.0)
    xg = x.clone().requires_grad_(True)
    y = F.gelu(xg, approximate="tanh")
    y.sum().backward()
    want = {"NONE": x, "ATOMIC": x + 3.0, "ADD": x + aux_before, "MUL": x * aux_before, "GELU": y.detach(), "GELU_DG": y.detach()}[epi]
    assert _rel_err(out.double(), want) < (1e-5 if f32 else 4e-3)
    if epi in ("GELU", "GELU_DG"):
        assert _rel_err(aux.double(), x if epi == "GELU" else xg.grad) < 4e-3
    buf[:Ma, 8:8 + N] = 3.0
    assert (buf == 3.0).all()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("M,N", [(128, 136), (256, 264), (304, 136)])
def test_gemm_sums_take_a_bias(a_mn, b_mn, M, N):
    """C += A B^T + bias, on both kernels and whatever the layout; grouped sums too. fp32 sums: K * 2^-24."""
    from innova_b200 import ops
    from innova_b200.ops import moe  # noqa: F401  (binds the grouped product)
    from innova_b200.ops import runtime as rt
    torch.manual_seed(3)
    dev, K = _dev(), 128
    A, B = torch.randn(M, K, device=dev).bfloat16(), torch.randn(N, K, device=dev).bfloat16()
    bias = torch.randn(N, device=dev).bfloat16() * 8
    out = torch.full((M, N), 2.0, device=dev)
    ops.gemm(A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B, out=out, a_mn=a_mn, b_mn=b_mn, epilogue=ops.EPI_ATOMIC, bias=bias, split_k=1)
    want = A.double() @ B.double().t() + bias.double() + 2.0
    assert _rel_err(out.double(), want) < 1e-5
    if a_mn and b_mn:
        off = torch.tensor([0, K], dtype=torch.int32, device=dev)
        out = torch.full((1, M, N), 2.0, device=dev)
        At, Bt = A.t().contiguous(), B.t().contiguous()
        rt.check(rt.lib().inv_gemm_grouped(At.data_ptr(), Bt.data_ptr(), out.data_ptr(), M, N, K, M, N, N, 1, 1, ops.EPI_ATOMIC, bias.data_ptr(), 0, 0, 0, 1, 1, 2,
                                           1, 0, off.data_ptr(), 0, 0, M * N, rt.status_tensor(dev).data_ptr(), rt.stream_ptr()), "inv_gemm_grouped")
        assert _rel_err(out[0].double(), want) < 1e-5


@pytest.mark.parametrize("M,F_,K,half,bias", [(129, 8, 64, 8, False), (300, 136, 72, 136, True), (257, 128, 200, 160, True), (1000, 1408, 512, 1408, False),
                                             (2 * 74 * 256 + 9, 392, 64, 400, True)])
def test_gemm_swiglu_matches_product_and_activation(M, F_, K, half, bias):
    """The product whose epilogue is the gated activation: ragged tiles, up rows further down than the gate's count, more tiles than pairs. Against
    fp64 of the projections rounded to bf16, which leaves the rounding of the result (2^-9) and projections that round the other way (2^-8)."""
    from innova_b200 import ops
    torch.manual_seed(11)
    dev = _dev()
    x = torch.randn(M, K + 8, device=dev).bfloat16()[:, :K]
    w = (torch.randn(half + F_, K, device=dev) * 0.2).bfloat16()
    b = torch.randn(half + F_, device=dev).bfloat16() if bias else None
    y = ops.gemm_swiglu(x, w, F_, half, b)
    z = x.double() @ w.double().t() + (0 if b is None else b.double())
    z = z.bfloat16().double()
    want = F.silu(z[:, :F_]) * z[:, half:]
    assert y.shape == (M, F_) and _rel_err(y.double(), want) < 2.0 ** -7
    if half == F_:
        two = ops.swiglu(ops.linear(x.contiguous(), w, b))
        assert _rel_err(y.double(), two.double()) < 2.0 ** -7
    assert ops.gemm_swiglu(x[:128], w, F_, half, b) is None and ops.gemm_swiglu(x.float(), w, F_, half, b) is None
    assert ops.gemm_swiglu(x[:, 1:], w[:, 1:], F_, half, b) is None


def test_gemm_wgrad_shape():
    """dW[N,K] += dY[T,N]^T X[T,K] with a long reduction and split-K chosen by the wrapper."""
    from innova_b200 import ops
    torch.manual_seed(2)
    dev = _dev()
    T, N, K = 4096, 768, 256
    dy = (torch.randn(T, N, device=dev) * 0.1).bfloat16()
    x = (torch.randn(T, K, device=dev) * 0.1).bfloat16()
    g = torch.zeros(N, K, device=dev, dtype=torch.float32)
    ops.gemm(dy, x, out=g, a_mn=True, b_mn=True, epilogue=ops.EPI_ATOMIC)
    assert _rel_err(g, dy.float().t() @ x.float()) < 1e-2


def test_linear_autograd():
    from innova_b200 import ops
    torch.manual_seed(3)
    dev = _dev()
    x = (torch.randn(4, 96, 256, device=dev) * 0.5).bfloat16().requires_grad_(True)
    w = (torch.randn(512, 256, device=dev) * 0.05).bfloat16().requires_grad_(True)
    b = torch.randn(512, device=dev).bfloat16().requires_grad_(True)
    y = ops.linear(x, w, b)
    gy = torch.randn_like(y)
    y.backward(gy)
    xr, wr, br = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True), b.detach().float().requires_grad_(True)
    yr = F.linear(xr, wr, br)
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 1e-2
    assert _rel_err(w.grad, wr.grad) < 1e-2
    assert _rel_err(b.grad, br.grad) < 1e-2


def test_mlp_gelu_autograd():
    from innova_b200 import ops
    torch.manual_seed(4)
    dev = _dev()
    T, E, Fh = 384, 256, 1024
    x = (torch.randn(T, E, device=dev) * 0.5).bfloat16().requires_grad_(True)
    res = torch.randn(T, E, device=dev).bfloat16().requires_grad_(True)
    w1 = (torch.randn(Fh, E, device=dev) * 0.05).bfloat16().requires_grad_(True)
    b1 = (torch.randn(Fh, device=dev) * 0.1).bfloat16().requires_grad_(True)
    w2 = (torch.randn(E, Fh, device=dev) * 0.05).bfloat16().requires_grad_(True)
    b2 = (torch.randn(E, device=dev) * 0.1).bfloat16().requires_grad_(True)
    y = ops.mlp_gelu(x, w1, b1, w2, b2, res)
    gy = torch.randn_like(y)
    y.backward(gy)
    ps = [t.detach().float().requires_grad_(True) for t in (x, res, w1, b1, w2, b2)]
    yr = F.linear(F.gelu(F.linear(ps[0], ps[2], ps[3]), approximate="tanh"), ps[4], ps[5]) + ps[1]
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2
    for t, r in zip((x, res, w1, b1, w2, b2), ps):
        assert _rel_err(t.grad, r.grad) < 2e-2


# ------------------------------------------------------------------------------------------ norms
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("T,D", [(64, 768), (333, 1024), (16, 5120), (100, 264)])
def test_norm(rms, T, D):
    from innova_b200 import ops
    torch.manual_seed(5)
    dev = _dev()
    x = torch.randn(T, D, device=dev).bfloat16().requires_grad_(True)
    g = (1 + 0.1 * torch.randn(D, device=dev)).bfloat16().requires_grad_(True)
    b = (0.1 * torch.randn(D, device=dev)).bfloat16().requires_grad_(True)
    y = ops.rms_norm(x, g, 1e-5) if rms else ops.layer_norm(x, g, b, 1e-5)
    gy = torch.randn_like(y)
    y.backward(gy)
    xr, gr, br = (t.detach().float().requires_grad_(True) for t in (x, g, b))
    if rms:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * gr
    else:
        yr = F.layer_norm(xr, (D,), gr, br, 1e-5)
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 2e-2
    assert _rel_err(g.grad, gr.grad) < 2e-2
    if not rms:
        assert _rel_err(b.grad, br.grad) < 2e-2


# ------------------------------------------------------------------------------------------ elementwise
def test_embedding_and_grad():
    from innova_b200 import ops
    torch.manual_seed(6)
    dev = _dev()
    V, D, B, S = 1000, 128, 3, 64
    wte = torch.randn(V, D, device=dev).bfloat16().requires_grad_(True)
    wpe = torch.randn(S, D, device=dev).bfloat16().requires_grad_(True)
    ids = torch.randint(0, V, (B, S), device=dev)
    ids[0, 0] = V + 5  # out of range -> row 0
    y = ops.embedding(ids, wte, wpe)
    gy = torch.randn_like(y)
    y.backward(gy)
    a, p = wte.detach().float().requires_grad_(True), wpe.detach().float().requires_grad_(True)
    safe = torch.where(ids < V, ids, torch.zeros_like(ids))
    yr = F.embedding(safe, a) + p[:S]
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(wte.grad, a.grad) < 1e-2
    assert _rel_err(wpe.grad, p.grad) < 1e-2


def test_activations():
    from innova_b200 import ops
    torch.manual_seed(7)
    dev = _dev()
    x = torch.randn(200, 512, device=dev).bfloat16().requires_grad_(True)
    y = ops.gelu(x)
    gy = torch.randn_like(y)
    y.backward(gy)
    xr = x.detach().float().requires_grad_(True)
    yr = F.gelu(xr, approximate="tanh")
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2 and _rel_err(x.grad, xr.grad) < 2e-2
    gu = torch.randn(200, 1024, device=dev).bfloat16().requires_grad_(True)
    y = ops.swiglu(gu)
    gy = torch.randn_like(y)
    y.backward(gy)
    gr = gu.detach().float().requires_grad_(True)
    g_, u_ = gr.chunk(2, -1)
    yr = F.silu(g_) * u_
    yr.backward(gy.float())
    assert _rel_err(y, yr) < 1e-2 and _rel_err(gu.grad, gr.grad) < 2e-2


def test_rope():
    from innova_b200 import ops
    torch.manual_seed(8)
    dev = _dev()
    B, S, H, Hkv, D = 2, 48, 4, 2, 64
    qkv = torch.randn(B, S, (H + 2 * Hkv) * D, device=dev).bfloat16()
    cos, sin = ops.rope_tables(128, D, 10000.0, dev)
    ref = ops.rope_qk(qkv.cpu().float(), cos.cpu(), sin.cpu(), H, Hkv, D)
    x = qkv.clone().requires_grad_(True)
    y = ops.rope_qk(x * 1.0, cos, sin, H, Hkv, D)
    assert _rel_err(y.cpu(), ref) < 1e-2
    gy = torch.randn_like(y)
    y.backward(gy)
    xr = qkv.cpu().float().requires_grad_(True)
    ops.rope_qk(xr, cos.cpu(), sin.cpu(), H, Hkv, D).backward(gy.cpu().float())
    assert _rel_err(x.grad.cpu(), xr.grad) < 1e-2


def test_cross_entropy():
    from innova_b200 import ops
    torch.manual_seed(9)
    dev = _dev()
    T, V, Vp = 300, 50257, 50304
    logits = (torch.randn(T, Vp, device=dev) * 2).bfloat16()
    labels = torch.randint(0, V, (T,), device=dev)
    labels[5] = -100
    lr = logits[:, :V].float().requires_grad_(True)
    ref = F.cross_entropy(lr, labels, ignore_index=-100)
    ref.backward()
    lg = logits.clone().requires_grad_(True)
    loss = ops.cross_entropy(lg * 1.0, labels, vocab=V)
    loss.backward()
    assert abs(float(loss) - float(ref)) < 2e-3 * max(1.0, abs(float(ref)))
    assert _rel_err(lg.grad[:, :V], lr.grad) < 2e-2
    assert float(lg.grad[:, V:].abs().max()) == 0.0


def test_lm_head_ce_fused():
    from innova_b200 import ops
    torch.manual_seed(10)
    dev = _dev()
    T, E, V, Vp = 640, 256, 1000, 1024
    x = (torch.randn(T, E, device=dev)).bfloat16().requires_grad_(True)
    w = (torch.randn(Vp, E, device=dev) * 0.05).bfloat16().requires_grad_(True)
    labels = torch.randint(0, V, (T,), device=dev)
    loss = ops.lm_head_cross_entropy(x, w, labels, vocab=V, chunk=256)
    loss.backward()
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = F.cross_entropy(F.linear(xr, wr)[:, :V], labels)
    ref.backward()
    assert abs(float(loss) - float(ref)) < 5e-3
    assert _rel_err(x.grad, xr.grad) < 3e-2
    assert _rel_err(w.grad[:V], wr.grad[:V]) < 3e-2


def test_adamw_matches_torch():
    from innova_b200.training.flat_engine import FlatParamEngine
    torch.manual_seed(11)
    dev = _dev()
    lin = torch.nn.Linear(96, 160).to(dev).bfloat16()
    ref = torch.nn.Linear(96, 160).to(dev).float()
    ref.load_state_dict({k: v.float() for k, v in lin.state_dict().items()})
    eng = FlatParamEngine(lin, lr=1e-2, weight_decay=0.1, max_grad_norm=0.0)
    opt = torch.optim.AdamW([{"params": [ref.weight], "weight_decay": 0.1}, {"params": [ref.bias], "weight_decay": 0.0}], lr=1e-2, eps=1e-8)
    for _ in range(5):
        gw, gb = torch.randn_like(ref.weight), torch.randn_like(ref.bias)
        lin.weight.main_grad.copy_(gw)
        lin.bias.main_grad.copy_(gb)
        ref.weight.grad, ref.bias.grad = gw.clone(), gb.clone()
        eng.step()
        opt.step()
    w_master = eng.master[: ref.weight.numel()].view_as(ref.weight)
    assert _rel_err(w_master, ref.weight) < 1e-4
    assert _rel_err(lin.weight, ref.weight) < 1e-2
    assert float(eng.flat_grad.abs().max()) == 0.0


def test_an_optimizer_step_is_captured_after_many():
    """The step's row of hyperparameters has been sent before by then; a capture permits no wait for that."""
    from innova_b200.training.flat_engine import FlatParamEngine
    dev = _dev()
    out = []
    for graph in (False, True):
        torch.manual_seed(4)
        lin = torch.nn.Linear(64, 64).to(dev).bfloat16()
        eng = FlatParamEngine(lin, lr=1e-2)
        grads = torch.randn(41, eng.total, device=dev)
        for g in grads[:40]:
            eng.flat_grad.copy_(g)
            eng.step()
        eng.flat_grad.copy_(grads[40])
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                eng.step()
            g.replay()
        else:
            eng.step()
        torch.cuda.synchronize()
        out.append(eng.master.clone())
    # the squares of the gradient norm are added in any order: 2^-23 of 41 steps of 1e-2, and as many roundings of values below one half
    assert torch.allclose(*out, rtol=0, atol=1e-6)


def test_optimizer_steps_beside_a_capture_on_another_thread():
    """More steps than rows of hyperparameters, on a stream of their own, while this thread captures: neither disturbs the other."""
    import threading
    from innova_b200.training.flat_engine import FlatParamEngine
    dev = _dev()
    torch.manual_seed(4)
    lin = torch.nn.Linear(64, 64).to(dev).bfloat16()
    eng = FlatParamEngine(lin, lr=1e-2)
    eng.step()
    x, y = torch.ones(64, device=dev), torch.empty(64, device=dev)
    errors, side = [], torch.cuda.Stream()

    def steps():
        try:
            with torch.cuda.stream(side):
                for _ in range(40):
                    eng.step()
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        torch.mul(x, 2.0, out=y)
        t = threading.Thread(target=steps)
        t.start()
        t.join()
        torch.add(y, 1.0, out=y)
    g.replay()
    torch.cuda.synchronize()
    assert not errors and eng.step_count == 41 and torch.equal(y, torch.full_like(y, 3.0))


# ------------------------------------------------------------------------------------------ attention
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,H,Hkv,causal", [(2, 256, 4, 4, True), (1, 384, 4, 2, True), (2, 200, 2, 2, True), (1, 256, 2, 1, False),
                                              (1, 1024, 2, 2, True)])
def test_flash_attention(D, B, S, H, Hkv, causal):
    from innova_b200 import ops
    torch.manual_seed(12)
    dev = _dev()
    qkv = (torch.randn(B, S, (H + 2 * Hkv) * D, device=dev) * 0.7).bfloat16().requires_grad_(True)
    out = ops.flash_attention(qkv, H, Hkv, D, causal=causal)
    go = torch.randn_like(out)
    out.backward(go)
    qr = qkv.detach().float().requires_grad_(True)
    ref = ops.attention_reference(qr, H, Hkv, D, causal=causal, scale=1.0 / math.sqrt(D))
    ref.backward(go.float())
    assert _rel_err(out, ref) < 2e-2
    dq, dk, dv = qkv.grad.split([H * D, Hkv * D, Hkv * D], dim=-1)
    rq, rk, rv = qr.grad.split([H * D, Hkv * D, Hkv * D], dim=-1)
    assert _rel_err(dv, rv) < 3e-2
    assert _rel_err(dk, rk) < 3e-2
    assert _rel_err(dq, rq) < 3e-2


# Persistent CTAs: several work items each, in both orders (by length, and head by head beyond twelve rounds), both forms for 128-wide heads.
# Items of a round: 296 forward (148 where 128-wide heads take one CTA an SM), 148 backward.
@pytest.mark.parametrize("D,B,S,H,Hkv,causal,window", [
    (64, 26, 333, 8, 8, True, 0), (64, 26, 333, 8, 4, True, 0), (64, 26, 333, 8, 4, False, 0), (64, 16, 640, 8, 8, True, 100), (64, 224, 200, 8, 8, True, 0),
    (128, 26, 333, 8, 4, True, 0), (128, 26, 333, 8, 8, False, 0), (128, 10, 1000, 8, 4, True, 0), (128, 13, 700, 8, 4, False, 0), (128, 8, 1100, 8, 8, True, 200),
    (128, 28, 900, 8, 2, True, 0), (128, 150, 130, 16, 8, True, 0)])
def test_flash_attention_over_many_items(D, B, S, H, Hkv, causal, window):
    """Outputs, statistics and gradients of every head of every sequence: what one item leaves behind for the next one on its CTA (barrier phases, Q, K and V
    loaded ahead, sums and statistics) would show in single heads. Bounds: those of the single-item tests, per head."""
    from innova_b200.ops.attention import _FlashAttnFn, attention_reference
    torch.manual_seed(S)
    dev = _dev()
    qkv = (torch.randn(B, S, (H + 2 * Hkv) * D, device=dev) * 0.7).bfloat16()

    class Ctx:
        def save_for_backward(self, *a):
            self.saved_tensors = a

    ctx = Ctx()
    out = _FlashAttnFn.forward(ctx, qkv, H, Hkv, D, causal, D ** -0.5, window)
    lse = ctx.saved_tensors[2]
    go = torch.randn_like(out)
    grad = _FlashAttnFn.backward(ctx, go)[0]

    def off(a, b, heads):                               # per sequence and head
        a, b = (x.float().reshape(-1, S, heads, D) for x in (a, b))
        return float(((a - b).norm(dim=(1, 3)) / b.norm(dim=(1, 3))).max())

    for b0 in range(0, B, 8):                           # a few sequences at a time: the reference keeps all scores
        sl = slice(b0, b0 + 8)
        qr = qkv[sl].float().requires_grad_(True)
        ref = attention_reference(qr, H, Hkv, D, causal=causal, scale=D ** -0.5, window=window)
        ref.backward(go[sl].float())
        n = ref.shape[0]
        q, k, _ = qr.detach().split([H * D, Hkv * D, Hkv * D], dim=-1)
        q, k = q.view(n, S, H, D).transpose(1, 2), k.view(n, S, Hkv, D).transpose(1, 2).repeat_interleave(H // Hkv, dim=1)
        z = q @ k.transpose(-1, -2) * D ** -0.5
        pos = torch.arange(S, device=dev)
        if causal:
            z = z.masked_fill(pos[None, :] > pos[:, None], float("-inf"))
        if window:
            z = z.masked_fill(pos[:, None] - pos[None, :] >= window, float("-inf"))
        # the kernel adds the exponentials as packed bf16 in fours: 2^-8 of the denominator, a hundredth of a power of two
        assert float((lse[sl] - torch.logsumexp(z, -1) * 1.4426950408889634).abs().max()) < 2e-2
        assert off(out[sl], ref, H) < 2e-2
        for a, r, heads in zip(grad[sl].split([H * D, Hkv * D, Hkv * D], dim=-1), qr.grad.split([H * D, Hkv * D, Hkv * D], dim=-1), (H, Hkv, Hkv)):
            assert off(a, r, heads) < 3e-2


# ------------------------------------------------------------------------------------------ model
@pytest.mark.parametrize("D,B,S,H,Hkv,window", [(64, 2, 1024, 4, 4, 256), (64, 1, 640, 4, 2, 100), (128, 1, 768, 4, 2, 300), (64, 1, 512, 2, 2, 33),
                                                 (64, 1, 384, 2, 1, 128)])
def test_sliding_window_attention(D, B, S, H, Hkv, window):
    """Causal local window in the tcgen05 flash kernels (forward and backward) against fp32 attention with the same mask:
    windows that end inside a key block, windows shorter than a block (rows that see nothing of their first block), GQA."""
    from innova_b200 import ops
    torch.manual_seed(11)
    dev = _dev()
    qkv = (torch.randn(B, S, (H + 2 * Hkv) * D, device=dev) * 0.5).bfloat16().requires_grad_(True)
    out = ops.flash_attention(qkv, H, Hkv, D, causal=True, window=window)
    ref_in = qkv.detach().float().requires_grad_(True)
    ref = ops.attention_reference(ref_in, H, Hkv, D, True, None, window)
    assert _rel_err(out, ref) < 2e-2
    w = torch.randn_like(ref)
    (out.float() * w).sum().backward()
    (ref * w).sum().backward()
    assert _rel_err(qkv.grad, ref_in.grad) < 3e-2
    from innova_b200.ops import runtime as rt
    rt.check_status()
    # memory-efficient attention routes the same pattern to these kernels
    from innova_b200.ops.mea import MEAConfig, MemoryEfficientAttention
    if S % 128 == 0:
        q, k, v = qkv.detach().split([H * D, Hkv * D, Hkv * D], -1)
        Q = q.view(B, S, H, D).transpose(1, 2).contiguous()
        K = k.view(B, S, Hkv, D).transpose(1, 2).contiguous()
        V = v.view(B, S, Hkv, D).transpose(1, 2).contiguous()
        mea = MemoryEfficientAttention(MEAConfig(use_block_sparse=True, block_sparse_window=window, causal=True))
        o2 = mea(Q, K, V).transpose(1, 2).reshape(B, S, H * D)
        assert _rel_err(o2, ref) < 2e-2


def test_dense_model_matches_cpu_reference():
    from innova_b200.models import DenseModel, gpt2_small
    torch.manual_seed(13)
    dev = _dev()
    cfg = gpt2_small(num_layers=2, hidden_size=256, num_heads=4, ffn_hidden_size=512, vocab_size=1000, max_seq_len=256)
    cpu = DenseModel(cfg, dtype=torch.float32)
    gpu = DenseModel(cfg, dtype=torch.bfloat16)
    gpu.load_state_dict({k: v.bfloat16() for k, v in cpu.state_dict().items()})
    gpu.to(dev)
    ids = torch.randint(0, 1000, (2, 256))
    labels = torch.randint(0, 1000, (2, 256))
    lc = cpu(ids, labels)
    lg = gpu(ids.to(dev), labels.to(dev))
    assert abs(float(lc) - float(lg)) < 3e-2
    lc.backward()
    lg.backward()
    for (n, pc), (_, pg) in zip(cpu.named_parameters(), gpu.named_parameters()):
        assert pg.grad is not None, n
        assert _rel_err(pg.grad.cpu(), pc.grad) < 8e-2, n


def test_llama_style_model_trains():
    from innova_b200.models import DenseModel, TransformerConfig
    from innova_b200.training.trainer import Trainer, TrainConfig
    torch.manual_seed(14)
    dev = _dev()
    cfg = TransformerConfig(vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, head_dim=64, ffn_hidden_size=512, num_kv_heads=2,
                            max_seq_len=128)
    model = DenseModel(cfg, dtype=torch.bfloat16, device=dev)
    tr = Trainer(model, TrainConfig(lr=2e-3))
    ids = torch.randint(0, 512, (4, 128), device=dev)
    labels = torch.roll(ids, -1, dims=1)
    first = float(tr.train_step(ids, labels))
    for _ in range(10):
        last = float(tr.train_step(ids, labels))
    assert last < first - 0.5


@pytest.mark.parametrize("N,K", [(136, 72), (264, 200), (520, 128)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_grouped_gemm_results_stay_in_their_groups(N, K, b_mn):
    """Products of expert segments (rows in multiples of 128, one segment empty, an unused tile) and their weight gradients, whose ragged matrices
    lie next to each other: every group's result, and nothing beside it. bf16 results carry one rounding; fp32 sums K or rows * 2^-24."""
    from innova_b200.ops import moe
    torch.manual_seed(5)
    dev = _dev()
    rows, E = [128, 0, 384, 256], 4
    offs = [0, 128, 128, 512, 768]
    R = 768 + 128                                                     # the last tile belongs to nobody
    tile = torch.tensor([0, 2, 2, 2, 3, 3, -1], dtype=torch.int32, device=dev)
    off = torch.tensor(offs, dtype=torch.int32, device=dev)
    x = torch.randn(R, K, device=dev).bfloat16()
    w = (torch.randn(E, N, K, device=dev) * 0.2).bfloat16()
    stack = w.transpose(1, 2).contiguous() if b_mn else w             # [E, K, N] or [E, N, K]
    buf = torch.full((R, N + 8), 7.0, dtype=torch.bfloat16, device=dev)
    out = buf[:, :N]
    moe._grouped(x, stack.view(-1, stack.shape[-1]), out, mode=1, E=E, tile_expert=tile, offsets=off, rows_b=stack.shape[1], b_mn=b_mn, M=R, N=N, K=K)
    for e in range(E):
        if rows[e]:
            assert _rel_err(out[offs[e]:offs[e + 1]].double(), x[offs[e]:offs[e + 1]].double() @ w[e].double().t()) < 4e-3
    assert (buf[768:] == 7.0).all() and (buf[:, N:] == 7.0).all()
    # weight gradients: C_e[K, N] += x_e^T dy_e
    dy = torch.randn(R, N, device=dev).bfloat16()
    g = torch.full((E, K, N), 2.0, device=dev)
    moe._grouped(x, dy, g, mode=2, E=E, tile_expert=None, offsets=off, rows_b=0, a_mn=True, b_mn=True, M=K, N=N, K=R, split_k=2, stride_c=K * N)
    for e in range(E):
        want = x[offs[e]:offs[e + 1]].double().t() @ dy[offs[e]:offs[e + 1]].double() + 2.0
        assert _rel_err(g[e].double(), want) < 1e-5

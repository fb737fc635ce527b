"""Block-32 codebook compute formats and the STE op (CPU arithmetic; the GPU kernel is checked against it)."""
import pytest
import torch

from innova_b200.ops import quant


def test_oil8_beats_oil4_beats_spark_and_codebook_training_helps():
    torch.manual_seed(0)
    w = torch.randn(64, 128) * 0.05
    snr = {}
    for fmt in ("oil8", "oil4", "spark", "oil1"):
        idx, sc, q = quant.quantize_blockwise(w, fmt, want_dequant=True)
        assert idx.numel() == w.numel() and sc.numel() == w.numel() // 32
        snr[fmt] = quant.snr_db(w, q)
        back = quant.dequantize_blockwise(idx, sc, fmt).view_as(w)
        assert torch.allclose(back, q, atol=1e-6)
    assert snr["oil8"] > snr["oil4"] > snr["spark"] > 0
    cb = quant.train_codebook(w, "oil4")
    assert cb.numel() == 16 and bool((cb[1:] >= cb[:-1]).all())
    _, _, q2 = quant.quantize_blockwise(w, "oil4", codebook=cb, want_dequant=True)
    assert quant.snr_db(w, q2) >= snr["oil4"] - 0.5
    cb2 = quant.ema_update_codebook(cb, w, decay=0.9)
    assert cb2.shape == cb.shape


def test_ste_gradient_is_identity_and_values_are_on_the_grid():
    torch.manual_seed(1)
    w = (torch.randn(8, 64) * 0.1).requires_grad_(True)
    q = quant.ste_fake_quant(w, "oil8")
    assert not torch.equal(q, w) and (q - w).abs().max() < 0.01
    g = torch.randn_like(q)
    q.backward(g)
    assert torch.equal(w.grad, g)
    # every block holds its abs-max exactly (codebook ends are -1 and +1)
    blk = w.detach().view(-1, 32)
    qb = q.detach().view(-1, 32)
    assert torch.allclose(qb.abs().amax(1), blk.abs().amax(1), atol=1e-7)


def test_nibble_packing():
    idx = torch.arange(32, dtype=torch.uint8) % 16
    p = quant.pack_nibbles(idx)
    assert p.numel() == 16 and int(p[0]) == (0 | (1 << 4)) and int(p[7]) == (14 | (15 << 4))


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["oil8", "oil4", "spark", "oil1"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gpu_kernel_matches_cpu_arithmetic(fmt, dtype):
    torch.manual_seed(2)
    w = (torch.randn(37, 100) * 0.07).to(dtype)
    idx_c, sc_c, q_c = quant.quantize_blockwise(w.float(), fmt, want_dequant=True)
    idx_g, sc_g, q_g = quant.quantize_blockwise(w.cuda(), fmt, want_dequant=True)
    assert torch.allclose(sc_g.cpu(), sc_c, rtol=1e-5, atol=1e-8)
    assert (idx_g.cpu() != idx_c).float().mean() < 0.01  # ties may flip
    assert torch.allclose(q_g.float().cpu(), q_c.view_as(w), atol=2e-3 if dtype == torch.bfloat16 else 1e-4)
    if fmt in ("oil8", "oil4"):
        back = quant.dequantize_blockwise(idx_g, sc_g, fmt)
        assert torch.allclose(back.float().cpu().view_as(w), q_c.view_as(w), atol=2e-3)
    wg = w.cuda().requires_grad_(True)
    out = quant.ste_fake_quant(wg, fmt)
    out.sum().backward()
    assert torch.equal(wg.grad, torch.ones_like(wg))


def test_quant_weight_cpu_linear():
    from innova_b200.ops.oil_linear import quantize_weight, oil_linear
    torch.manual_seed(3)
    w = torch.randn(48, 128) * 0.05
    x = torch.randn(5, 128)
    for fmt, tol in (("oil8", 0.02), ("oil4", 0.15)):
        qw = quantize_weight(w, fmt)
        assert qw.nbytes() < w.numel() * (0.6 if fmt == "oil4" else 1.1)
        y = oil_linear(x, qw)
        ref = x @ w.t()
        assert float((y - ref).norm() / ref.norm()) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["oil4", "oil8"])
@pytest.mark.parametrize("M,N,K", [(64, 768, 4096), (1, 256, 128), (200, 1000, 1344), (300, 128, 64), (64, 384, 2752), (128, 2048, 512), (128, 256, 128), (100, 640, 192)])
def test_gpu_oil_gemm_matches_dequantised_matmul(fmt, M, N, K):
    from innova_b200.ops import runtime as rt
    from innova_b200.ops.oil_linear import quantize_weight, oil_linear
    torch.manual_seed(4)
    dev = torch.device("cuda", 0)
    w = (torch.randn(N, K, device=dev) * 0.05)
    x = torch.randn(M, K, device=dev).bfloat16()
    bias = torch.randn(N, device=dev).bfloat16()
    res = torch.randn(M, N, device=dev).bfloat16()
    qw = quantize_weight(w, fmt, bias=bias)
    y = oil_linear(x, qw, residual=res)
    rt.check_status()
    ref = x.float() @ qw.dequantize().float().t() + bias.float() + res.float()
    assert float((y.float() - ref).norm() / ref.norm()) < 1e-2
    y2 = oil_linear(x, qw, residual=res)  # the accumulator was left clean
    assert torch.equal(y, y2) or float((y2.float() - ref).norm() / ref.norm()) < 1e-2


def _codes_and_values(qw):
    """What dequantize() says with plain PyTorch calls."""
    shifts = {"oil4": (0, 4), "oil8": (0,)}.get(qw.fmt, (0, 2, 4, 6))
    mask = {"oil4": 15, "oil8": 255}.get(qw.fmt, 3)
    codes = torch.stack([(qw.idx >> s) & mask for s in shifts], -1).view(qw.N, qw.K)
    vals = qw.codebook[codes.long()].bfloat16()
    return codes, (vals.view(qw.N, -1, 32) * qw.scales.view(qw.N, -1, 1)).view(qw.N, qw.K)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fmt", ["oil4", "oil8", "spark", "oil1"])
@pytest.mark.parametrize("n", [32, 7 * 32, 8 * 32, 9 * 32, 300 * 32 + 5, 148 * 8 * 64 * 32 + 64])
def test_gpu_whole_blocks_and_single_values_quantise_alike(n, fmt, dtype):
    """The kernel of whole blocks against the one that takes a value per lane (any address), bit for bit: uneven codebooks,
    blocks of zeros, values that are no numbers or too large, the last block cut short."""
    g = torch.Generator(device="cuda").manual_seed(n % 1000)
    w = torch.randn(n, device="cuda", generator=g) * 0.02
    w[:32] = 0.0
    if n > 200:
        w[40], w[70], w[100], w[101] = float("nan"), float("inf"), -1e30, 1e-38
    w = w.to(dtype)
    off = torch.empty(n + 1, dtype=dtype, device="cuda")[1:].copy_(w)          # not on a 16-byte boundary
    K = {"oil4": 16, "oil8": 256}.get(fmt, 16)
    uneven = torch.linspace(-1, 1, K, device="cuda").pow(3).contiguous()
    for cb in (None, uneven) if fmt in ("oil4", "oil8") else (None,):
        a, b = quant.quantize_blockwise(w, fmt, cb, want_dequant=True), quant.quantize_blockwise(off, fmt, cb, want_dequant=True)
        for x, y in zip(a, b):
            assert torch.equal(torch.nan_to_num(x.float(), 7.0), torch.nan_to_num(y.float(), 7.0))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fmt", ["oil4", "oil8", "spark", "oil1"])
@pytest.mark.parametrize("N,K", [(1, 64), (3, 192), (128, 4096), (1001, 320)])
def test_gpu_quantised_matrix_and_back(N, K, fmt, dtype):
    from innova_b200.ops.oil_linear import quantize_weight
    w = (torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N)) * 0.02).to(dtype)
    qw = quantize_weight(w, fmt)
    idx, sc, _ = quant.quantize_blockwise(w, fmt)
    codes, values = _codes_and_values(qw)
    assert torch.equal(codes, idx.view(N, K)) and torch.equal(qw.scales, sc.view(N, -1).bfloat16())
    assert torch.equal(qw.dequantize(), values)
    off = torch.empty(N * K + 1, dtype=dtype, device="cuda")[1:].copy_(w.view(-1)).view(N, K)
    assert torch.equal(quantize_weight(off, fmt).idx, qw.idx)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["oil4", "oil8", "spark"])
@pytest.mark.parametrize("M,N,K", [(1, 32000, 4096), (64, 22016, 4096), (64, 4096, 11008), (100, 6144, 4096), (128, 4096, 4096)])
def test_gpu_oil_gemm_ring_of_index_tiles_wraps(fmt, M, N, K):
    """More index tiles per CTA than the ring holds, the weights warm in L2 from the second call on: a tile must not be replaced
    before it has been used. The operands are exact in bf16 and the sums fp32, so the error is the rounding of the result (2^-9)."""
    from innova_b200.ops import runtime as rt
    from innova_b200.ops.oil_linear import quantize_weight, oil_linear
    g = torch.Generator(device="cuda").manual_seed(8)
    qw = quantize_weight(torch.randn(N, K, device="cuda", generator=g) * 0.02, fmt)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    ref = x.float() @ qw.dequantize().float().t()
    for _ in range(4):
        y = oil_linear(x, qw).float()
        assert float((y - ref).norm() / ref.norm()) < 2.0 ** -8
    rt.check_status()


def test_fused_finish_fallbacks_cpu():
    from innova_b200 import ops
    from innova_b200.ops.oil_linear import oil_linear, oil_linear_norm, oil_linear_swiglu, quantize_weight
    torch.manual_seed(5)
    w = torch.randn(64, 128) * 0.05
    x = torch.randn(3, 128)
    qw = quantize_weight(w, "oil4")
    assert torch.allclose(oil_linear_swiglu(x, qw), ops.swiglu(oil_linear(x, qw)))
    res = torch.randn(3, 64)
    nw = torch.rand(64) + 0.5
    y, h = oil_linear_norm(x, qw, res, nw, 1e-5)
    assert torch.allclose(y, oil_linear(x, qw, res))
    assert torch.allclose(h, ops.rms_norm(y, nw, 1e-5))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 64, 200])
def test_gpu_fused_finish_matches_unfused(M):
    from innova_b200 import ops
    from innova_b200.ops import runtime as rt
    from innova_b200.ops.oil_linear import oil_linear, oil_linear_norm, oil_linear_swiglu, quantize_weight
    torch.manual_seed(6)
    dev = torch.device("cuda", 0)
    K, N = 512, 768
    x = torch.randn(M, K, device=dev).bfloat16()
    qw = quantize_weight(torch.randn(N, K, device=dev) * 0.05, "oil4", bias=torch.randn(N, device=dev).bfloat16() * 0.1)
    a = oil_linear_swiglu(x, qw)
    b = ops.swiglu(oil_linear(x, qw))
    assert float((a.float() - b.float()).abs().max()) <= 2e-2 * float(b.float().abs().max())
    res = torch.randn(M, N, device=dev).bfloat16()
    nw = (torch.rand(N, device=dev) + 0.5).bfloat16()
    y, h = oil_linear_norm(x, qw, res, nw, 1e-5)
    y_ref = oil_linear(x, qw, res)
    h_ref = ops.rms_norm(y_ref, nw, 1e-5)
    rt.check_status()
    assert float((y.float() - y_ref.float()).abs().max()) <= 2e-2 * float(y_ref.float().abs().max())
    assert float((h.float() - h_ref.float()).abs().max()) <= 3e-2 * float(h_ref.float().abs().max())
    # the accumulator is left clean by every finish variant
    assert torch.equal(oil_linear(x, qw, res), y_ref) or float((oil_linear(x, qw, res).float() - y_ref.float()).abs().max()) < 1e-1


def test_ste_quantizer_static_codebook_and_mixed_blocks():
    from innova_b200.ops.quant import STEQuantizer, default_codebook
    STEQuantizer.reset_static_codebooks()
    torch.manual_seed(0)
    q = STEQuantizer()
    w1 = torch.randn(4096) * 0.02
    y1 = q(w1, "oil4")
    cb = q.codebook(w1, "oil4")
    assert cb.numel() == 16 and not torch.allclose(cb, default_codebook("oil4"))          # trained on the first tensor
    w2 = torch.rand(4096)                                                                   # another distribution: same codebook
    q(w2, "oil4")
    assert q.codebook(w2, "oil4") is cb
    # the trained codebook fits the first tensor better than the uniform grid the training started from
    from innova_b200.ops.quant import ste_fake_quant
    assert (y1 - w1).square().mean() < (ste_fake_quant(w1, "oil4", codebook=torch.linspace(-1.0, 1.0, 16)) - w1).square().mean()
    w = (torch.randn(1024) * 0.1).requires_grad_(True)
    fm = ["oil8", "oil4", "spark", "fp32"]
    y = q.forward_mixed(w, fm, block=256)
    err = [(y[i * 256:(i + 1) * 256] - w[i * 256:(i + 1) * 256]).detach().square().mean().item() for i in range(4)]
    assert err[3] == 0.0 and err[0] < err[1] < err[2]
    y.sum().backward()
    assert torch.equal(w.grad, torch.ones_like(w))                                          # identity gradient through every format
    assert STEQuantizer(use_ste=False)(w, "oil4") is w
    STEQuantizer.reset_static_codebooks()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["oil4", "oil8", "spark", "oil1"])
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (1, 3072, 2048), (3, 1000, 192), (8, 24, 5632), (9, 2048, 1344), (16, 11264, 2048), (7, 4096, 11008),
                                   (13, 40, 128), (16, 5000, 5056)])
def test_gpu_few_tokens_one_launch(fmt, M, N, K):
    """The skinny product against fp64 on the same bf16 operands, in its three forms, with the norm in front and without. Its sums are
    fp32, so what is left is the rounding of the results (2^-9) and, with the norm, of the normed row (another 2^-9)."""
    from innova_b200.ops.functional import rms_norm
    from innova_b200.ops.oil_linear import (SKINNY_SUMS, SKINNY_SWIGLU, _skinny, oil_linear, oil_linear_norm, oil_linear_swiglu, quantize_weight)
    g = torch.Generator(device="cuda").manual_seed(M * 7 + K)
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    qw = quantize_weight(torch.randn(N, K, device="cuda", generator=g) * 0.05, fmt, bias=bias)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    nw = torch.randn(K, device="cuda", generator=g).bfloat16()
    w = qw.dequantize().double()

    def off(y, ref):
        return float((y.double() - ref).norm() / ref.norm())

    def out(n, dtype=torch.bfloat16):
        return torch.full((M, n), float("nan"), dtype=dtype, device="cuda")

    prod = x.double() @ w.t()
    plain = prod + bias.double() + res.double()
    y = _skinny(x, qw, out(N), residual=res)
    assert off(y, plain) < 2.0 ** -8 and torch.equal(y, _skinny(x, qw, out(N), residual=res))
    assert off(_skinny(x, qw, out(N, torch.float32), SKINNY_SUMS), prod) < 1e-5
    gate, up = (prod + bias.double()).bfloat16().double().chunk(2, -1)
    glu = torch.nn.functional.silu(gate) * up
    assert off(_skinny(x, qw, out(N // 2), SKINNY_SWIGLU), glu) < 2.0 ** -7
    normed = rms_norm(x, nw, 1e-5).double() @ w.t()
    assert off(_skinny(x, qw, out(N, torch.float32), SKINNY_SUMS, norm=(nw, 1e-5)), normed) < 2.0 ** -8
    nwo = torch.randn(N, device="cuda", generator=g).bfloat16()
    assert off(oil_linear(x, qw, residual=res), plain) < 2.0 ** -8 and off(oil_linear_swiglu(x, qw), glu) < 2.0 ** -7
    y, hn = oil_linear_norm(x, qw, res, nwo, 1e-5)
    assert off(y, plain) < 2.0 ** -8 and off(hn, rms_norm(y, nwo, 1e-5).double()) < 2.0 ** -8


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 5, 16, 17])
@pytest.mark.parametrize("N,offset", [(20, 0), (100, 4), (256, 4), (256, 0)])
def test_gpu_projection_and_norm_of_widths_and_weights_off_16_bytes(M, N, offset):
    """Widths that are a multiple of four only, and norm weights on 8 bytes, with few tokens as with more; the results carry no graph."""
    from innova_b200.ops.oil_linear import oil_linear_norm, quantize_weight
    g = torch.Generator(device="cuda").manual_seed(N + M)
    qw = quantize_weight(torch.randn(N, 128, device="cuda", generator=g) * 0.1, "oil4")
    x, res = (torch.randn(M, n, device="cuda", generator=g).bfloat16() for n in (128, N))
    nw = torch.nn.Parameter(torch.randn(N + offset, device="cuda", generator=g).bfloat16()[offset:])
    y, h = oil_linear_norm(x, qw, res, nw, 1e-5)
    want = x.double() @ qw.dequantize().double().t() + res.double()
    normed = y.double() * torch.rsqrt(y.double().square().mean(-1, keepdim=True) + 1e-5) * nw.detach().double()
    assert not y.requires_grad and not h.requires_grad
    assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -8 and float((h.double() - normed).norm() / normed.norm()) < 2.0 ** -8


@pytest.mark.gpu
@pytest.mark.parametrize("M,fits", [(1, 73728), (8, 11008), (9, 9728), (16, 5632)])
def test_gpu_few_tokens_up_to_the_limit_of_shared_memory(M, fits):
    """The longest rows that the skinny product takes at a token count, the next longer ones (the tile product's) and a token too many."""
    from innova_b200.ops import runtime as rt
    from innova_b200.ops.oil_linear import SKINNY_SUMS, _skinny, oil_linear, quantize_weight, skinny_takes
    g = torch.Generator(device="cuda").manual_seed(M)
    for K in (fits, fits + 256):
        qw = quantize_weight(torch.randn(40, K, device="cuda", generator=g) * 0.05, "oil4")
        x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        want = x.double() @ qw.dequantize().double().t()
        assert skinny_takes(qw, M) == (K == fits) and not skinny_takes(qw, 17)
        assert float((oil_linear(x, qw).double() - want).norm() / want.norm()) < 2.0 ** -8
    with pytest.raises(RuntimeError):
        _skinny(x, qw, torch.empty(M, 40, device="cuda"), SKINNY_SUMS)
    rt.check_status()

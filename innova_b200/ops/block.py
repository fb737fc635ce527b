"""A pre-norm transformer block as one autograd function: every launch of its forward pass, and every launch of its backward pass, is issued
by one native call (csrc/block_program.cu). The kernels, their arguments and their order are those of the layers one by one
(``ops.norm_residual``, ``linear``, ``rope_qk``, ``flash_attention``, ``mlp_gelu`` / ``swiglu``, ``ste_fake_quant``), so the results are the same;
what goes is 20 us of Python, autograd and binding per launch, which bounds a training step below a few thousand tokens.

Reference behaviour covered: TransformerBlock::forward (src/transformer.cpp:380-409) and its autograd (src/autograd_grad.cpp).
"""
from __future__ import annotations

import ctypes as C
import functools
import importlib
import struct

import torch

from .. import _native
from . import runtime as rt
from .gemm import main_grad_of, main_grads
from .quant import BLOCK, MODES, default_codebook

_gemm = importlib.import_module(".gemm", __package__)      # the module: the package exports the function under this name

_native.register_cuda_sigs({"inv_block_fwd": [_native.vp], "inv_block_bwd": [_native.vp], "inv_block_bytes": [_native.i32] + [_native.i64] * 9 + [_native.vp],
                              "inv_block_split_k": [_native.i64] * 3})

# BlockDesc: 12 parameters, tables, positions, codebook, x, y, saved, status, stream | dy, dx, two column sums, 12 gradients, scratch | 14 sizes |
# eps1, eps2, scale
_PACK = struct.Struct("=12Q 9Q 17Q 14q 3d").pack
_FORWARD_ONLY = (0,) * 17


SAVED, SCRATCH, FORWARD = 0, 1, 2


@functools.lru_cache(maxsize=256)
def _bytes(which, B, S, E, H, Hkv, D, F, gated, quantised):
    """What the native side lays out: the forward pass's buffer when a backward pass follows, that pass's scratch, a forward pass's alone."""
    n = C.c_long()
    if rt.lib().inv_block_bytes(which, B, S, E, H, Hkv, D, F, gated, quantised, C.addressof(n)) != 0:
        raise ValueError("block sizes")
    return n.value


def _ptr(t):
    return 0 if t is None else t.data_ptr()


class _BlockFn(torch.autograd.Function):
    """params: norm 1 (gamma, beta), qkv (weight, bias), o (weight, bias), norm 2, first and second product of the MLP; biases and beta may
    be None."""

    @staticmethod
    def forward(ctx, x, cfg, keep, cos, sin, positions, codebook, *params):
        H, Hkv, D, F, gated, rms, eps1, eps2, mode = cfg
        B, S, E = x.shape
        dev = x.device
        # without gradients nothing is left for a backward pass, and buffers share their places
        saved = torch.empty(_bytes(SAVED if keep else FORWARD, B, S, E, H, Hkv, D, F, gated, int(codebook is not None)), dtype=torch.uint8, device=dev)
        y = torch.empty_like(x)
        _issue("inv_block_fwd", cfg, (B, S, E), params, cos, sin, positions, codebook, x, y.data_ptr(), saved, _FORWARD_ONLY, int(keep))
        if not keep:
            return y
        ctx.cfg = cfg
        ctx.main_grads = main_grads(*params)
        ctx.save_for_backward(x, saved, cos, sin, positions, codebook, *params)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, saved, cos, sin, positions, codebook, *params = ctx.saved_tensors
        H, Hkv, D, F, gated = ctx.cfg[:5]
        B, S, E = x.shape
        dev = x.device
        dy = dy.contiguous()
        colsum = rt.take_colsum(dy.view(-1, E))
        # fp32 gradients: the parameter's main_grad, or a buffer of zeros that goes back to autograd
        grads, out, ptrs = [], [], []
        for p, kept in zip(params, ctx.main_grads):
            if p is None:
                out.append(None)
                ptrs.append(0)
                continue
            mg = main_grad_of(p, kept)
            own = mg is not None and mg.is_contiguous() and mg.dtype == torch.float32
            g = mg if own else torch.zeros(p.shape, dtype=torch.float32, device=dev)
            if not own:
                grads.append((len(out), g, mg, p))
            out.append(None)
            ptrs.append(g.data_ptr())
        dx = torch.empty_like(x)
        dx_colsum = torch.empty(E, dtype=torch.float32, device=dev) if E <= 1024 else None
        scratch = torch.empty(_bytes(SCRATCH, B, S, E, H, Hkv, D, F, gated, int(codebook is not None)), dtype=torch.uint8, device=dev)
        _issue("inv_block_bwd", ctx.cfg, (B, S, E), params, cos, sin, positions, codebook, x, 0, saved,
               (dy.data_ptr(), dx.data_ptr(), _ptr(colsum), _ptr(dx_colsum), *ptrs, scratch.data_ptr()))
        if dx_colsum is not None:
            rt.offer_colsum(dx.view(-1, E), dx_colsum)
        for i, g, mg, p in grads:
            if mg is not None:
                mg.add_(g.view(mg.shape))
            else:
                out[i] = g.to(p.dtype)
        return (dx, None, None, None, None, None, None, *out)


def _issue(what, cfg, shape, params, cos, sin, positions, codebook, x, y, saved, backward, keep=1):
    H, Hkv, D, F, gated, rms, eps1, eps2, mode = cfg
    desc = _PACK(*[_ptr(p) for p in params], _ptr(cos), _ptr(sin), _ptr(positions), _ptr(codebook), x.data_ptr(), y, saved.data_ptr(),
                 rt.status_tensor(x.device).data_ptr(), rt.stream_ptr(), *backward,
                 *shape, H, Hkv, D, F, gated, rms, 0 if codebook is None else codebook.numel(), mode, int(codebook is not None), _gemm._kernel_select, keep,
                 eps1, eps2, D ** -0.5)
    n = getattr(rt.lib(), what)(desc)
    rt.check(min(n, 0), what)
    rt.count_launches(n - 1)


def _plain(t):
    return t is None or (type(t) in (torch.nn.Parameter, torch.Tensor) and t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous())


def block_forward(blk, x, rope, positions):
    """The block's output, or None where its layers have to run one by one: anything but bf16 on the GPU in plain, contiguous tensors; hooks, adapters
    or replaced parts inside the block; parameters of which only some want gradients; a collective that rides in the products' grids; tracing.
    Looked at in every call."""
    cfg, att, ffn, n1, n2 = blk.cfg, blk.attention, blk.ffn, blk.attention_norm, blk.ffn_norm
    gated = ffn.gated
    if (x.dim() != 3 or not _plain(x) or x.numel() == 0 or cfg.use_parallel_residual or ffn.adapter is not None
            or not (gated or cfg.activation == "gelu") or cfg.head_dim not in (64, 128) or _gemm._side_job_provider is not None
            or (cfg.ste_format and (cfg.ste_format not in MODES or cfg.ste_block != BLOCK)) or n1.kind != n2.kind):
        return None
    if torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.nn.modules.module._has_any_global_hook():
        return None
    first = ffn.gate_up_proj if gated else ffn.up_proj
    shifts = n1.kind == "layernorm"                     # an RMS norm has no use for a bias
    params = (n1.weight, n1.bias if shifts else None, att.qkv_proj.weight, att.qkv_proj.bias, att.o_proj.weight, att.o_proj.bias, n2.weight,
              n2.bias if shifts else None, first.weight, first.bias, ffn.down_proj.weight, ffn.down_proj.bias)
    grad = torch.is_grad_enabled()
    for p in params:
        if not _plain(p) or (grad and p is not None and not p.requires_grad):
            return None
    E, F, W = x.shape[2], ffn.down_proj.weight.shape[1], (cfg.num_heads + 2 * cfg.kv_heads) * cfg.head_dim
    if (params[2].shape != (W, E) or params[4].shape != (E, cfg.num_heads * cfg.head_dim) or params[8].shape != (2 * F if gated else F, E)
            or params[10].shape != (E, F) or n1.weight.shape[0] != E or n2.weight.shape[0] != E or E % 8 or F % 8):
        return None
    cos = sin = None
    if rope is not None:
        cos, sin = rope
        if cos.dtype != torch.float32 or not (cos.is_contiguous() and sin.is_contiguous()):
            return None
    codebook, mode = None, 0
    if cfg.ste_format:
        codebook = getattr(cfg, "ste_codebook", None)
        if codebook is None:
            codebook = default_codebook(cfg.ste_format, x.device)
        mode = MODES[cfg.ste_format]
    return _BlockFn.apply(x, (cfg.num_heads, cfg.kv_heads, cfg.head_dim, F, int(gated), int(n1.kind != "layernorm"), float(n1.eps), float(n2.eps), mode),
                          grad, cos, sin, positions, codebook, *params)

"""Causal self-attention (MHA / GQA / MQA) over a fused qkv buffer.

The raw entry points take the fused projection ``qkv[B*S, (Hq + 2*Hkv)*hd]`` and return
``out[B*S, Hq*hd]``.  On CUDA, bf16 forward and backward run on the tcgen05 flash kernels at any sequence length and
any head size up to 256 that is a multiple of 8: up to 128 in ``csrc/attention_flash.cu``, above that and soft-capped scores
in ``csrc/attention_wide.cu``.  Other head sizes up to 256 are zero-padded to the next multiple of 8 (``padded_shape``):
padded head columns add nothing to any dot product.  On CPU a plain softmax(QK^T)V restatement is used, which is also the
oracle for tests.  The library attention is reached only for other dtypes or when forced with ``ZEN_ATTN=lib``.
"""
from __future__ import annotations

import ctypes
import functools
import os

import torch
import torch.nn.functional as F

from .. import _native

_MODE = os.environ.get("ZEN_ATTN", "auto")        # auto | own | lib


def kernel_covers(seq, hq, hkv, hd, dtype) -> bool:
    """Shapes the tcgen05 attention kernels handle: head sizes up to 256 (multiples of 8) at any sequence length."""
    return dtype == torch.bfloat16 and hq % hkv == 0 and hd <= 256 and hd % 8 == 0


def have_kernel(seq, hq, hkv, hd, dtype) -> bool:
    """True when forward and backward run on the hand-written kernels for this shape, soft-capped or not."""
    return _MODE != "lib" and kernel_covers(seq, hq, hkv, hd, dtype)


def padded_shape(seq, hq, hkv, hd, dtype):
    """(seq', hd') of the covered shape that (seq, hd) is zero-padded to, or None when padding cannot help."""
    if _MODE == "lib" or dtype != torch.bfloat16 or hq % hkv or hd > 256:
        return None
    return seq, (hd + 7) // 8 * 8


def pad_qkv(qkv, bsz, seq, nheads, hd, seq_p, hd_p):
    """[B*S, nheads*hd] -> zero-padded [B*S', nheads*hd'] (contiguous)."""
    out = qkv.new_zeros(bsz, seq_p, nheads, hd_p)
    out[:, :seq, :, :hd] = qkv.view(bsz, seq, nheads, hd)
    return out.view(bsz * seq_p, nheads * hd_p)


def unpad(t, bsz, seq, nheads, hd, seq_p, hd_p):
    return t.view(bsz, seq_p, nheads, hd_p)[:, :seq, :, :hd].reshape(bsz * seq, nheads * hd)


def attention_fwd_kernel(qkv, bsz, seq, hq, hkv, hd, scale, softcap: float = 0.0):
    """tcgen05 forward: returns (out[B*S, Hq*hd], lse2[B, Hq, S rounded up to 128]) with lse2 in base 2 of the scaled scores.
    ``softcap`` > 0 soft-caps the scaled scores, cap * tanh(s / cap), before the softmax (Gemma-2)."""
    assert qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.stride(1) == 1
    out = torch.empty(bsz * seq, hq * hd, dtype=qkv.dtype, device=qkv.device)
    lse2 = torch.empty(bsz, hq, (seq + 127) // 128 * 128, dtype=torch.float32, device=qkv.device)
    if hd <= 128 and softcap <= 0:
        rc = _native.lib().zen_flash_fwd(_native.ptr(qkv), _native.ptr(out), _native.ptr(lse2), bsz, seq, hq, hkv, hd,
                                         qkv.stride(0), out.stride(0), float(scale), _native.stream_ptr())
        _native.check(rc, "zen_flash_fwd")
        return out, lse2
    rc = _native.lib().zen_attn_fwd(_native.ptr(qkv), _native.ptr(out), _native.ptr(lse2), bsz, seq, hq, hkv, hd,
                                    qkv.stride(0), out.stride(0), float(scale), float(softcap),
                                    _native.stream_ptr())
    _native.check(rc, "zen_attn_fwd")
    return out, lse2


@functools.lru_cache(maxsize=4096)
def _flash_ds_bytes(bsz, seq, hq, hd) -> int:
    """Bytes of scratch for which the backward keeps dS between its kernels, or 0."""
    out = ctypes.c_int64()
    _native.lib().zen_flash_ds_bytes(bsz, seq, hq, hd, ctypes.addressof(out))
    return out.value


def scratch(most: int, least: int, device) -> tuple:
    """(bytes, 1) of size ``most``, or (bytes, 0) of size ``least`` where the device has no room for as much: what dS takes between the
    kernels of the backward is up to 3 GB, and a step that fits without it has to run."""
    if most > least:
        try:
            return torch.empty(most, dtype=torch.uint8, device=device), 1
        except torch.OutOfMemoryError:
            pass
    return torch.empty(least, dtype=torch.uint8, device=device), 0


def attention_bwd_kernel(dout, qkv, out, lse2, bsz, seq, hq, hkv, hd, scale, softcap: float = 0.0):
    """tcgen05 backward: gradient of the fused qkv buffer (no atomics)."""
    dout = dout if (dout.is_contiguous() and dout.data_ptr() % 16 == 0) else dout.contiguous()
    dqkv = torch.empty_like(qkv)
    if hd <= 128 and softcap <= 0:
        need, nstat = _flash_ds_bytes(bsz, seq, hq, hd), 8 * lse2.numel()
        temp, keep_ds = scratch(nstat + need, nstat, qkv.device)                                 # row statistics (a multiple of 1 KB), dS
        stat = temp.data_ptr()
        rc = _native.lib().zen_flash_bwd(qkv.data_ptr(), out.data_ptr(), dout.data_ptr(), lse2.data_ptr(), stat, dqkv.data_ptr(), bsz, seq, hq,
                                         hkv, hd, qkv.stride(0), out.stride(0), dqkv.stride(0), float(scale), stat + nstat if keep_ds else 0,
                                         _native.stream_ptr())
        if rc:
            _native.check(rc, "zen_flash_bwd")
        return dqkv
    stat = torch.empty(2, *lse2.shape, dtype=torch.float32, device=qkv.device)
    # few KV heads (MQA / GQA): the query heads of a group are shared out over several CTA pairs
    hsplit, part = _native.lib().zen_attn_hsplit(bsz, seq, hq, hkv, hd), None
    if hsplit > 1:
        part = torch.empty(2 * hsplit * bsz * seq * hkv * hd, dtype=torch.float32, device=qkv.device)
    rc = _native.lib().zen_attn_bwd(_native.ptr(qkv), _native.ptr(out), _native.ptr(dout), _native.ptr(lse2), _native.ptr(stat),
                                    _native.ptr(dqkv), bsz, seq, hq, hkv, hd, qkv.stride(0), out.stride(0), dqkv.stride(0),
                                    float(scale), float(softcap), _native.ptr(part), hsplit,
                                    _native.stream_ptr())
    _native.check(rc, "zen_attn_bwd")
    return dqkv


def attention_error() -> int:
    lib = _native.lib()
    return int(lib.zen_attn_error()) or int(lib.zen_flash_error())


def _split(qkv, bsz, seq, hq, hkv, hd):
    t = qkv.view(bsz, seq, hq + 2 * hkv, hd)
    q = t[:, :, :hq].transpose(1, 2)
    k = t[:, :, hq:hq + hkv].transpose(1, 2)
    v = t[:, :, hq + hkv:].transpose(1, 2)
    return q, k, v


def reference_attention(qkv, bsz, seq, hq, hkv, hd, scale, softcap: float = 0.0):
    q, k, v = _split(qkv.float(), bsz, seq, hq, hkv, hd)
    rep = hq // hkv
    k = k.repeat_interleave(rep, dim=1)
    v = v.repeat_interleave(rep, dim=1)
    s = (q @ k.transpose(-1, -2)) * scale
    if softcap > 0:
        s = softcap * torch.tanh(s / softcap)
    mask = torch.ones(seq, seq, dtype=torch.bool, device=qkv.device).tril()
    s = s.masked_fill(~mask, float("-inf"))
    o = torch.softmax(s, -1) @ v
    return o.transpose(1, 2).reshape(bsz * seq, hq * hd).to(qkv.dtype)


def attention_fwd(qkv, bsz, seq, hq, hkv, hd, scale, softcap: float = 0.0):
    if not qkv.is_cuda:
        return reference_attention(qkv, bsz, seq, hq, hkv, hd, scale, softcap), ()
    if have_kernel(seq, hq, hkv, hd, qkv.dtype) and qkv.is_contiguous():
        out, lse2 = attention_fwd_kernel(qkv, bsz, seq, hq, hkv, hd, scale, softcap)
        return out, (lse2,)
    if softcap > 0:
        return reference_attention(qkv, bsz, seq, hq, hkv, hd, scale, softcap), ()
    q, k, v = _split(qkv, bsz, seq, hq, hkv, hd)
    o = F.scaled_dot_product_attention(q, k, v, is_causal=True, scale=scale, enable_gqa=(hq != hkv))
    return o.transpose(1, 2).reshape(bsz * seq, hq * hd), ()


def attention_bwd(dout, qkv, out, saved, bsz, seq, hq, hkv, hd, scale, softcap: float = 0.0):
    """Gradient w.r.t. the fused qkv buffer: the tcgen05 kernels when the forward saved its statistics, else a
    recomputation under autograd."""
    if len(saved) == 1 and qkv.is_cuda:
        return attention_bwd_kernel(dout, qkv, out, saved[0], bsz, seq, hq, hkv, hd, scale, softcap)
    with torch.enable_grad():
        x = qkv.detach().requires_grad_(True)
        if not qkv.is_cuda or softcap > 0:
            o = reference_attention(x, bsz, seq, hq, hkv, hd, scale, softcap)
        else:
            q, k, v = _split(x, bsz, seq, hq, hkv, hd)
            o = F.scaled_dot_product_attention(q, k, v, is_causal=True, scale=scale, enable_gqa=(hq != hkv))
            o = o.transpose(1, 2).reshape(bsz * seq, hq * hd)
        (g,) = torch.autograd.grad(o, x, dout)
    return g

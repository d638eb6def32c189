"""A decoder block as one autograd node whose forward and backward are one native call each (csrc/block.cu).

Same kernels and the same numbers as the op-by-op path in ``models/decoder.py``; what goes is the host time between the
launches.  Taken for bf16 CUDA blocks without tensor parallelism or checkpointing whose shapes the attention kernels cover
(``usable``); everything else stays op by op.
"""
from __future__ import annotations

import ctypes
import math

import torch

from .. import _native
from . import attention as A
from . import autograd as O
from . import gemm as G

# order of the parameters in the native structures
PARAMS = ("norm1_w", "norm1_b", "norm2_w", "norm2_b", "postnorm1_w", "postnorm2_w", "qkv_w", "qkv_b", "o_w", "o_b", "up_w", "up_b",
          "down_w", "down_b")
_PROJ_W = (6, 8, 10, 12)                     # qkv, attention out, up, down
_NORM_PAIRS = ((0, 1), (2, 3))


class _Pick(ctypes.Structure):
    _fields_ = [("kind", ctypes.c_int32), ("p0", ctypes.c_int32), ("p1", ctypes.c_int32), ("pad", ctypes.c_int32)]


class _Block(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_int32) for n in ("d", "hq", "hkv", "hd", "inner", "layer_norm", "unit_offset", "act_mode", "gated", "rope",
                                               "w_in_out")]
                + [(n, ctypes.c_float) for n in ("eps", "theta", "scale", "softcap")] + [("pad", ctypes.c_int32)]
                + [("w", ctypes.c_void_p * 14), ("fwd", _Pick * 4), ("dx", _Pick * 4), ("dw", _Pick * 4),
                   ("fwd_only", _Pick * 4)])


class _Grads(ctypes.Structure):
    _fields_ = [("g", ctypes.c_void_p * 14), ("acc", ctypes.c_int32 * 14)]


class _Workspace(ctypes.Structure):
    _fields_ = [("ws", ctypes.c_void_p), ("n_ws", ctypes.c_uint64), ("cnt", ctypes.c_void_p), ("n_cnt", ctypes.c_int32), ("pad", ctypes.c_int32)]


def _pick(plan) -> _Pick:
    kind, *how = plan
    return _Pick({"one": 0, "pair": 1, "cluster": 2}[kind], how[0], how[1] if len(how) > 1 else 0, 0)


def _pick_weight(M: int, N: int, K: int) -> _Pick:
    return _Pick(3, 0, 0, 0) if G.groups(M, N) else _pick(G._plan(M, N, K, 0))


_workspaces: dict = {}


def _workspace(device) -> int:
    """Address of the GEMM workspace description of the current stream."""
    key = (device.index, _native.stream_ptr())
    w = _workspaces.get(key)
    if w is None:
        ws, n_ws, cnt, n_cnt = G._workspace_args(device)
        w = _workspaces[key] = _Workspace(ws, n_ws, cnt, n_cnt, 0)
    return ctypes.addressof(w)


class _Plan:
    """The native description of one block for one (batch, sequence) and the sizes of its buffers."""

    def __init__(self, blk, params, bsz, seq):
        cfg = blk.cfg
        lib = _native.lib()
        assert lib.zen_block_size() == ctypes.sizeof(_Block) and lib.zen_block_grads_size() == ctypes.sizeof(_Grads), "block layout mismatch"
        d, hd, T = cfg.hidden_size, cfg.head_dim, bsz * seq
        z = _Block()
        z.d, z.hq, z.hkv, z.hd, z.inner = d, blk.hq, blk.hkv, hd, blk.inner
        z.layer_norm, z.unit_offset = int(cfg.layer_norm), int(cfg.norm_unit_offset)
        z.act_mode, z.gated = {"gelu_tanh": 0, "relu": 1, "swiglu": 2, "geglu": 3}[cfg.act], int(cfg.gated)
        z.rope, z.w_in_out = int(not cfg.learned_positions), int(cfg.weight_layout == "in_out")
        z.eps, z.theta, z.scale, z.softcap = cfg.norm_eps, cfg.rope_theta, 1.0 / math.sqrt(hd), cfg.attn_softcap
        for i, p in enumerate(params):
            z.w[i] = p.data_ptr() if p is not None else None
        q, h, u = (blk.hq + 2 * blk.hkv) * hd, blk.hq * hd, blk.inner * (2 if cfg.gated else 1)
        for i, (fin, fout) in enumerate(((d, q), (h, d), (d, u), (blk.inner, d))):
            z.fwd[i], z.dx[i] = _pick(G._plan(T, fout, fin, 0)), _pick(G._plan(T, fin, fout, 0))
            z.fwd_only[i] = _pick(G.plan_forward_only(T, fout, fin))
            z.dw[i] = _pick_weight(fin, fout, T) if z.w_in_out else _pick_weight(fout, fin, T)
        self.z, self.addr = z, ctypes.addressof(z)
        sizes = (ctypes.c_int64 * 5)()
        lib.zen_block_bytes(self.addr, bsz, seq, sizes)
        self.saved, self.saved_res, self.fwd_temp, self.bwd_temp, self.bwd_temp_least = (int(v) for v in sizes)


def usable(blk, x: torch.Tensor, bsz: int, seq: int) -> bool:
    """Whether ``blk`` (a ``models.decoder.Block``) runs natively on this input."""
    cfg = blk.cfg
    hd = cfg.head_dim
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2) or cfg.grad_checkpoint:
        return False
    if not (G.native_defaults() and A._MODE != "lib" and O._FUSE_ACT_COLSUM):
        return False
    if cfg.hidden_size % 8 or blk.inner % 8 or hd % 8 or not A.have_kernel(seq, blk.hq, blk.hkv, hd, x.dtype):
        return False
    return not (cfg.sliding_window and seq > cfg.sliding_window)


def _plan_for(blk, params, bsz, seq) -> _Plan:
    """The plan for the parameters as they are now: asked for in the forward and again in the backward, between which a
    parameter may have been given other storage (``p.data = ...``, a move to another device and back)."""
    key = [bsz, seq]
    for p in params:
        if p is not None:
            # not part of what is cached: another tensor may have come to lie at the same address
            if p.dtype is not torch.bfloat16 or not p.is_contiguous():
                raise ValueError("block parameters must be contiguous bf16 tensors")
            key.append(p.data_ptr())
    cached = blk.__dict__.get("_native_plan")
    if cached is None or cached[0] != key:
        if any(at % 16 for at in key[2:]):
            raise ValueError("block parameters must be 16-byte aligned")
        cached = blk.__dict__["_native_plan"] = (key, _Plan(blk, params, bsz, seq))
    return cached[1]


class BlockFn(torch.autograd.Function):
    """(dn, h2) = block(x, res).  ``tracked``: the parameters whose gradients travel through autograd; empty when every gradient
    is written straight into the reducer's bucket views (the node then has no edge to any parameter)."""

    @staticmethod
    def forward(ctx, x, res, blk, params, bsz, seq, claimed, recorded, *tracked):
        plan = _plan_for(blk, params, bsz, seq)
        x = x if x.is_contiguous() else x.contiguous()
        if res is not None and not res.is_contiguous():
            res = res.contiguous()
        dev = x.device
        saved = torch.empty(plan.saved_res if res is not None else plan.saved, dtype=torch.uint8, device=dev)
        temp = torch.empty(plan.fwd_temp, dtype=torch.uint8, device=dev)
        dn, h2 = torch.empty_like(x), torch.empty_like(x)
        rc = _native.lib().zen_block_fwd(plan.addr, bsz, seq, x.data_ptr(), _native.ptr(res), saved.data_ptr(), temp.data_ptr(), dn.data_ptr(),
                                         h2.data_ptr(), int(recorded), _workspace(dev), _native.stream_ptr())
        if rc:
            _native.check(rc, "zen_block_fwd")
        if claimed:
            for p in params:
                if p is not None:
                    p.zen_expected += 1
        ctx.save_for_backward(x, res, h2, saved, *[p for p in params if p is not None])
        ctx.args = (blk, params, bsz, seq, claimed, ctx.needs_input_grad[8:])
        ctx.set_materialize_grads(False)
        return dn, h2

    @staticmethod
    def backward(ctx, d_dn, d_h2):
        x, res, h2, saved, *_ = ctx.saved_tensors          # also checks that no parameter was changed in place since
        blk, params, bsz, seq, claimed, needs = ctx.args
        plan = _plan_for(blk, params, bsz, seq)
        dev = x.device
        if d_dn is None:
            d_dn = torch.zeros_like(x)
        elif not d_dn.is_contiguous():
            d_dn = d_dn.contiguous()
        if d_h2 is not None and not d_h2.is_contiguous():
            d_h2 = d_h2.contiguous()
        gr = _Grads()
        grads = []
        if claimed:
            for i, p in enumerate(params):
                if p is not None:
                    gr.g[i] = p.grad.data_ptr()
                    gr.acc[i] = not p.zen_fresh
                    p.zen_fresh = False
        else:
            it = iter(needs)
            for i, p in enumerate(params):
                if p is None:
                    continue
                g = torch.empty_like(p) if next(it) else None
                grads.append(g)
                if g is not None:
                    gr.g[i] = g.data_ptr()
        dx = torch.empty_like(x)
        temp, keep_ds = A.scratch(plan.bwd_temp, plan.bwd_temp_least, dev)
        rc = _native.lib().zen_block_bwd(plan.addr, bsz, seq, x.data_ptr(), _native.ptr(res), h2.data_ptr(), saved.data_ptr(), temp.data_ptr(),
                                         keep_ds, d_dn.data_ptr(), _native.ptr(d_h2), dx.data_ptr(), ctypes.addressof(gr), _workspace(dev),
                                         _native.stream_ptr())
        if rc:
            _native.check(rc, "zen_block_bwd")
        if claimed:
            for p in reversed(params):
                if p is not None:
                    p.zen_ready(p)
        return (dx, dx if res is not None else None, None, None, None, None, None, None, *grads)


def run(blk, x, res, bsz: int, seq: int):
    own = blk._parameters                                  # attribute access would go through Module.__getattr__, 14 times
    params = [own[n] if n in own else getattr(blk, n) for n in PARAMS]
    present = [p for p in params if p is not None]
    recorded = torch.is_grad_enabled()
    claimed = False
    if recorded and x.requires_grad:
        claimed = all(p.requires_grad and getattr(p, "zen_direct_grad", False) and (g := p.grad) is not None and g.dtype == torch.bfloat16
                      and g.is_contiguous() for p in present)
    return BlockFn.apply(x, res, blk, params, bsz, seq, claimed, recorded, *(() if claimed else present))

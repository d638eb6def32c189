"""GEMM entry points.  bf16 CUDA operands run the tcgen05 kernels (csrc/gemm_tcgen05_2cta.cu, gemm_tcgen05.cu,
gemm_splitk.cu, chosen per shape by ``_plan``); everything else (CPU, fp32) runs ``torch.matmul`` and doubles as the
oracle in tests.

Naming: ``nt`` = A[M,K] @ B[N,K]^T, ``nn`` = A[M,K] @ B[K,N], ``tn`` = A[K,M]^T @ B[K,N].  These are the
forward, input-gradient and weight-gradient products of a linear layer (in either weight layout), so
no operand is ever transposed in memory.
"""
from __future__ import annotations

import ctypes
import functools
import os

import torch

from .. import _native

_FORCE_TORCH = os.environ.get("ZEN_GEMM", "") == "torch"
_PAIR_MODE = os.environ.get("ZEN_GEMM_2CTA", "auto")      # auto | 0 | 1


_clusters_cached = [0]


def _clusters() -> int:
    """CTA pairs the device runs at once (one per two SMs; 74 on a B200)."""
    if not _clusters_cached[0]:
        n = 148
        if torch.cuda.is_available():
            n = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
        _clusters_cached[0] = max(1, n // 2)
    return _clusters_cached[0]


# Time model of the kernels in microseconds, fitted to measurements on a B200 with cold caches (M 64 to 1 500, N 768 to
# 16 384, K 64 to 10 240): launch and epilogue, plus per round of output tiles and 64-wide block of K what one tile's
# pipeline takes, plus the store of every round after the first.  Only its order matters; it is within 15 % of the measured
# times over that range.
#   kernel          tile     CTAs a round   start   per round and block   per further round
_T_ONE128 = (128, 128, 148, 11.6, 0.22, 1.0)
_T_ONE256 = (128, 256, 148, 13.2, 0.38, 1.5)
_T_PAIR = (256, 256, 74, 13.0, 0.306, 1.0)
_TAIL_ROUND = 0.75                  # a last round whose tiles run as two halves of their columns
_SPLIT_EXCHANGE = 5.0               # two K slices of the pair kernel meeting through the workspace
_CLUSTER_START = 13.0               # csrc/gemm_splitk.cu: launch, cluster barriers and the sum over shared memory
# CTAs that clusters of up to 8 are sure to get side by side: with 132 and more, a second wave starts (18 -> 31 us measured
# at 144), since the GPCs' SM counts are not multiples of the cluster size
_CLUSTER_CTAS = 128


def _tiles(M, N, bm, bn):
    return ((M + bm - 1) // bm) * ((N + bn - 1) // bn)


def _t_one(M, N, nkb, k):
    bm, bn, per, start, step, store = k
    rounds = -(-_tiles(M, N, bm, bn) // per)
    return start + rounds * nkb * step + (rounds - 1) * store


def _t_pair(M, N, nkb):
    bm, bn, _, start, step, store = _T_PAIR
    per = _clusters()
    full, rem = divmod(_tiles(M, N, bm, bn), per)
    tail = 0.0 if rem == 0 else (_TAIL_ROUND if 2 * rem <= per else 1.0)
    return start + (full + tail) * nkb * step + max(0, full - (rem == 0)) * store


def use_pair_kernel(M: int, N: int, K: int) -> bool:
    """CTA-pair (256 x 256 tile) kernel rather than the single-CTA one, by the time model."""
    if _PAIR_MODE == "0":
        return False
    if _PAIR_MODE == "1":
        return M >= 256 and N >= 128
    if M < 129 or N < 129:
        return False
    nkb = (K + 63) // 64
    return _t_pair(M, N, nkb) < min(_t_one(M, N, nkb, _T_ONE128), _t_one(M, N, nkb, _T_ONE256))


def cluster_split(M: int, N: int, K: int) -> tuple[int, int, float]:
    """(tile columns, K slices, modelled time) of the cluster split-K kernel, slices 1 when it does not apply: as many slices
    as fit beside each other, at least four blocks of K in each; between 64- and 128-wide tiles the one that allows more."""
    nkb = (K + 63) // 64
    best = (128, 1, float("inf"))
    for bn in (64, 128):
        s = min(8, _CLUSTER_CTAS // _tiles(M, N, 128, bn), nkb // 4)
        if s >= 2 and s > best[1]:
            best = (bn, s, _CLUSTER_START + -(-nkb // s) * _T_ONE128[4])
    return best


_SPLITK = os.environ.get("ZEN_GEMM_SPLITK", "auto")       # auto | 0
_TAIL_SPLIT = os.environ.get("ZEN_GEMM_TAILSPLIT", "1") != "0"
_WS_FLOATS = 74 * 2 * 128 * 256                            # one fp32 partial tile per CTA of one full wave
_N_COUNTERS = 4096
_ws_cache: dict = {}
# below this K the extra pass over the partial tiles costs more than the idle clusters
_SPLITK_MIN_K = int(os.environ.get("ZEN_GEMM_SPLITK_MIN_K", "4096"))


def split_k_choice(M: int, N: int, K: int) -> int:
    """Number of K slices for the CTA-pair kernel, or 1.  Splitting pays when the output has far fewer 256 x 256
    tiles than the 74 clusters and K is long: the weight-gradient products of a transformer layer."""
    if _SPLITK == "0" or _PAIR_MODE == "0" or M < 256 or N < 256 or K < _SPLITK_MIN_K:
        return 1
    tm, tn = (M + 255) // 256, (N + 255) // 256
    tiles = tm * tn
    # both slices of every tile must be resident in the launch's single wave of clusters (they wait for each other)
    if (M * N) / (tiles * 65536.0) < 0.75 or tiles * 2 > _clusters():
        return 1
    splits = min(_clusters() // tiles, (K // 64) // 8, 2)  # two slices: the fast store path of the kernel
    return splits if splits >= 2 and tiles * splits * 2 * 128 * 256 <= _WS_FLOATS and tiles * 16 <= _N_COUNTERS else 1


def _splitk_workspace(device):
    """fp32 partial tiles and arrival counters for the split-K kernel, one pair per device and stream: the
    kernel's slices meet through them, so two launches may share them only in stream order."""
    key = (device.index, _native.stream_ptr())
    w = _ws_cache.get(key)
    if w is None:
        w = (torch.empty(_WS_FLOATS, dtype=torch.float32, device=device),
             torch.zeros(_N_COUNTERS, dtype=torch.int32, device=device))
        _ws_cache[key] = w
    return w


_ws_args: dict = {}


def _workspace_args(device) -> tuple:
    """(workspace address, floats, counters address, counters) of the current stream."""
    key = (device.index, _native.stream_ptr())
    v = _ws_args.get(key)
    if v is None:
        ws, cnt = _splitk_workspace(device)
        v = _ws_args[key] = (ws.data_ptr(), ws.numel(), cnt.data_ptr(), cnt.numel())
    return v


def _use_kernel(a: torch.Tensor, b: torch.Tensor) -> bool:
    return (a.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and not _FORCE_TORCH)


def _rowmajor(t: torch.Tensor) -> torch.Tensor:
    """2-D view with unit inner stride, 16-byte aligned base and row stride a multiple of 8."""
    if t.dim() != 2:
        t = t.reshape(-1, t.shape[-1])
    if t.stride(1) != 1 or t.stride(0) % 8 or t.data_ptr() % 16 or (t.shape[0] > 1 and t.stride(0) < t.shape[1]):
        cols = t.shape[1]
        pad = (-cols) % 8
        t = torch.nn.functional.pad(t, (0, pad))[:, :cols] if pad else t.contiguous()
    return t


@functools.lru_cache(maxsize=4096)
def _plan(M: int, N: int, K: int, bn: int):
    """Which kernel runs C[M, N] with depth K: ("pair", K slices), ("cluster", tile columns, K slices) or ("one", tile columns,
    0 = chosen by the launcher).  ``bn`` 128 / 256 / 512 forces the single-CTA tile width or the pair kernel."""
    if bn:
        return ("pair", 1) if bn == 512 else ("one", bn)
    nkb = (K + 63) // 64
    cbn, cs, ct = cluster_split(M, N, K) if _PAIR_MODE == "auto" and _SPLITK != "0" else (128, 1, float("inf"))
    splits = split_k_choice(M, N, K)
    if splits > 1:
        if ct < _T_PAIR[3] + _SPLIT_EXCHANGE + -(-nkb // splits) * _T_PAIR[4]:
            return ("cluster", cbn, cs)
        return ("pair", splits)
    pair = use_pair_kernel(M, N, K)
    t = _t_pair(M, N, nkb) if pair else min(_t_one(M, N, nkb, _T_ONE128), _t_one(M, N, nkb, _T_ONE256))
    if ct < t:
        return ("cluster", cbn, cs)
    if pair:
        return ("pair", 1)
    return ("one", 256 if _t_one(M, N, nkb, _T_ONE256) < _t_one(M, N, nkb, _T_ONE128) else 128)


@functools.lru_cache(maxsize=4096)
def plan_forward_only(M: int, N: int, K: int):
    """The plan for the products of a block that no backward will follow (scoring, validation).  K is cut into two at most, in two
    places: by ``split_k_choice`` (from 256 rows, K from 4096, tiles for at most half of the CTA pairs), and, K from 1024, in the
    last round of an output of at least 512 rows whose tiles fill 60 % of the pairs' rounds.  Never among the clusters of
    csrc/gemm_splitk.cu, nor in the last round of smaller outputs, which a third element 1 marks.

    So the order of summation is that of the products as they were before clusters shared K, but it is not the same at every
    token count: 3072 columns of depth 8192 take two slices at 256, 400 and 512 tokens and none at 300, 777 and 1024.  Another
    order moves one bf16 result in 600, which the layers after it amplify to the rounding noise of the whole computation.  After
    four layers the logits of 37 tokens differ by 1.27 % (Llama), 0.77 % (GPT-2) and 0.94 % (Gemma-2) between this plan and
    ``_plan``, and both are 1.50 %, 0.81 % and 1.00 % from fp32: neither is the more precise, and the same holds from 64 to 1024
    tokens.  This one leaves the results of scoring where they were."""
    splits = split_k_choice(M, N, K)
    if splits > 1:
        return ("pair", splits)
    nkb = (K + 63) // 64
    tiles = _tiles(M, N, 256, 256)
    fill = tiles / (-(-tiles // _clusters()) * _clusters()) * (M * N) / (tiles * 65536.0)
    if M >= 512 and N >= 256 and fill >= 0.6 and _PAIR_MODE != "0":
        return ("pair", 1)
    whole = (256, 256, _clusters()) + _T_PAIR[3:]
    if _PAIR_MODE != "0" and M > 128 and N > 128 and _t_one(M, N, nkb, whole) < min(_t_one(M, N, nkb, _T_ONE128), _t_one(M, N, nkb, _T_ONE256)):
        return ("pair", 1, 1)
    return ("one", 256 if _t_one(M, N, nkb, _T_ONE256) < _t_one(M, N, nkb, _T_ONE128) else 128)


def _launch(a, b, M, N, K, a_mn, b_mn, bias, out, accumulate, out_dtype, bn, pad_ok=False, last=False):
    a2, b2 = _rowmajor(a), _rowmajor(b)
    if out is None:
        out = torch.empty(M, N, dtype=out_dtype or torch.bfloat16, device=a.device)
        accumulate = False
    ldc = out.stride(0)
    fp32 = out.dtype == torch.float32
    assert out.dim() == 2 and out.shape == (M, N) and out.stride(1) == 1
    assert fp32 or out.dtype == torch.bfloat16
    if bias is not None:
        assert bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.numel() == N
    lib = _native.lib()
    kind, *how = _plan(M, N, K, bn)
    c = out.data_ptr()
    pbias = 0 if bias is None else bias.data_ptr()
    stream = _native.stream_ptr()
    if kind == "cluster" and c % 16:
        kind, how = "one", (0,)
    if kind == "pair":
        n_store = min((N + 7) // 8 * 8, ldc) if pad_ok and how[0] == 1 else 0
        if not _TAIL_SPLIT:
            lib.zen_gemm2_tail_split(0)
        ws, n_ws, cnt, n_cnt = _workspace_args(a.device) if _TAIL_SPLIT or how[0] > 1 else (0, 0, 0, 0)       # where K slices meet
        rc = lib.zen_gemm_bf16_2cta_splitk(a2.data_ptr(), b2.data_ptr(), c, pbias, M, N, K, a2.stride(0), b2.stride(0), ldc, a_mn,
                                           b_mn, fp32, bool(accumulate), how[0], ws, n_ws, cnt, n_cnt, n_store, bool(last), stream)
    elif kind == "cluster":
        rc = lib.zen_gemm_bf16_cluster_splitk(a2.data_ptr(), b2.data_ptr(), c, pbias, M, N, K, a2.stride(0), b2.stride(0), ldc, a_mn,
                                              b_mn, fp32, bool(accumulate), how[0], how[1], stream)
    else:
        rc = lib.zen_gemm_bf16(a2.data_ptr(), b2.data_ptr(), c, pbias, M, N, K, a2.stride(0), b2.stride(0), ldc, a_mn, b_mn, fp32,
                               bool(accumulate), how[0], stream)
    if rc:
        _native.check(rc, f"gemm ({kind})")
    return out


def gemm_nt(a, b, bias=None, out=None, accumulate=False, out_dtype=None, bn=0, pad_ok=False, last=False):
    """a[M,K] @ b[N,K]^T (+ bias[N]).  ``pad_ok``: ``out`` is the first N columns of a wider buffer whose columns up to
    the next multiple of 8 may be overwritten (with zeros); lets an odd N use the full-line store path.
    ``last``: no product reads the result (logits), so that it may be summed in whichever order is fastest."""
    M, K = a.shape[-2] if a.dim() == 2 else a.numel() // a.shape[-1], a.shape[-1]
    N = b.shape[0]
    if not _use_kernel(a, b):
        r = a.reshape(-1, K).float() @ b.float().t()
        return _finish(r, bias, out, accumulate, out_dtype or a.dtype)
    return _launch(a, b, M, N, K, False, False, bias, out, accumulate, out_dtype, bn, pad_ok, last)


def makes_loss_statistics(a, b) -> bool:
    """Whether :func:`gemm_nt_loss` runs for these operands: the CTA-pair kernel with whole K, on operands that need no copy."""
    if not _use_kernel(a, b) or a.dim() != 2 or b.dim() != 2 or _rowmajor(a) is not a or _rowmajor(b) is not b:
        return False
    kind, slices = _plan(a.shape[0], b.shape[0], a.shape[1], 0)[:2]
    return kind == "pair" and slices == 1


def gemm_nt_loss(a, b, labels, out=None, softcap: float = 0.0):
    """The logits a[M,K] @ b[N,K]^T as bf16 into ``out`` (the first N columns of a buffer whose rows are a multiple of 8 wide; None:
    nowhere) and what a cross-entropy against ``labels`` (int64) needs of them: ``(part, target)`` for ``elementwise.xent_finish``.
    Operands as :func:`makes_loss_statistics` asks."""
    (M, K), N = a.shape, b.shape[0]
    if labels.numel() != M or labels.dtype is not torch.int64 or not labels.is_contiguous() or labels.device != a.device:
        raise ValueError(f"{labels.numel()} labels of {labels.dtype} on {labels.device} for {M} rows of logits on {a.device}")
    part = torch.empty(2 * ((N + 255) // 256), (M + 31) // 32 * 32, 2, dtype=torch.float32, device=a.device)
    target = torch.empty(M, dtype=torch.float32, device=a.device)
    c, ldc = (0, 0) if out is None else (out.data_ptr(), out.stride(0))
    rc = _native.lib().zen_gemm_bf16_2cta_loss(a.data_ptr(), b.data_ptr(), c, M, N, K, a.stride(0), b.stride(0), ldc,
                                               min((N + 7) // 8 * 8, ldc), labels.data_ptr(), part.data_ptr(), part.shape[1],
                                               target.data_ptr(), float(softcap), _native.stream_ptr())
    _native.check(rc, "zen_gemm_bf16_2cta_loss")
    return part, target


def gemm_nn(a, b, bias=None, out=None, accumulate=False, out_dtype=None, bn=0):
    """a[M,K] @ b[K,N] (+ bias[N])."""
    K = a.shape[-1]
    M = a.numel() // K
    N = b.shape[1]
    if not _use_kernel(a, b):
        r = a.reshape(-1, K).float() @ b.float()
        return _finish(r, bias, out, accumulate, out_dtype or a.dtype)
    return _launch(a, b, M, N, K, False, True, bias, out, accumulate, out_dtype, bn)


def gemm_tn(a, b, out=None, accumulate=False, out_dtype=None, bn=0):
    """a[K,M]^T @ b[K,N]: the weight-gradient product (sum over tokens)."""
    M, N = a.shape[-1], b.shape[-1]
    K = a.numel() // M
    if not _use_kernel(a, b):
        r = a.reshape(-1, M).float().t() @ b.reshape(-1, N).float()
        return _finish(r, None, out, accumulate, out_dtype or a.dtype)
    return _launch(a, b, M, N, K, True, True, None, out, accumulate, out_dtype, bn)


# ---------------------------------------------------------------------------------------------------------------
# Deferred weight gradients.  The weight-gradient products of a transformer layer are small (27 / 9 / 36 / 36 output
# tiles for GPT-2 small against 74 CTA pairs) and nothing downstream in backward waits for them, so a linear layer's
# backward may queue its product here instead of launching it; GROUP_SIZE queued products (or the end of the backward
# pass, or an explicit flush) go out as ONE launch whose clusters walk the tiles of all of them.
class _GemmDesc(ctypes.Structure):
    _fields_ = [("A", ctypes.c_void_p), ("B", ctypes.c_void_p), ("C", ctypes.c_void_p),
                ("M", ctypes.c_int32), ("N", ctypes.c_int32), ("K", ctypes.c_int32),
                ("lda", ctypes.c_int32), ("ldb", ctypes.c_int32), ("ldc", ctypes.c_int32),
                ("out_fp32", ctypes.c_int32), ("accumulate", ctypes.c_int32)]


GROUP_SIZE = int(os.environ.get("ZEN_GEMM_GROUP", "4"))      # 0 / 1 = launch every weight gradient by itself
_pending: list = []
_callback_armed = [False]


def groups(M: int, N: int) -> bool:
    """Whether a weight gradient of this shape shares a grouped launch.  Products with many tiles fill the clusters by
    themselves; grouping them only delays their gradient."""
    return GROUP_SIZE > 1 and _PAIR_MODE != "0" and M >= 256 and N >= 256 and _tiles(M, N, 256, 256) <= 2 * _clusters()


def native_defaults() -> bool:
    """No switch of this module asks for another path than the one csrc/block.cu takes."""
    return GROUP_SIZE > 1 and _PAIR_MODE == "auto" and _TAIL_SPLIT and not _FORCE_TORCH


def defer_tn(a, b, out, accumulate: bool, done=None) -> None:
    """Queue ``out (+)= a[K,M]^T @ b[K,N]`` (bf16 CUDA operands, ``out`` a 2-D bf16 / fp32 tensor with unit inner stride);
    ``done()`` runs right after the launch that contains it has been enqueued.  Falls back to an immediate
    :func:`gemm_tn` when grouping is off or the operands do not qualify."""
    M, N = a.shape[-1], b.shape[-1]
    K = a.numel() // M
    ok = (groups(M, N) and _use_kernel(a, b) and out.is_cuda and out.dim() == 2 and out.stride(1) == 1 and out.dtype in (torch.bfloat16, torch.float32))
    if not ok:
        gemm_tn(a, b, out=out, accumulate=accumulate)
        if done is not None:
            done()
        return
    if any(item[2].data_ptr() == out.data_ptr() for item in _pending):
        flush_deferred()                           # two products into one output never share a launch
    a2, b2 = _rowmajor(a), _rowmajor(b)
    _pending.append((a2, b2, out, M, N, K, bool(accumulate), done))
    arm_flush_at_end_of_backward()
    if len(_pending) >= GROUP_SIZE:
        flush_deferred()


def arm_flush_at_end_of_backward() -> bool:
    """Ask the autograd engine to call :func:`flush_deferred` when the running backward pass ends.  False when no
    backward pass is running (the caller then flushes, or does not defer)."""
    if not _callback_armed[0]:
        try:
            torch.autograd.Variable._execution_engine.queue_callback(flush_deferred)
            _callback_armed[0] = True
        except RuntimeError:
            return False
    return True


def flush_deferred() -> None:
    """Launch whatever :func:`defer_tn` has queued (one launch per GROUP_SIZE products) and run the callbacks."""
    _callback_armed[0] = False
    while _pending:
        batch = _pending[:min(max(GROUP_SIZE, 1), _native.lib().zen_gemm_group_max())]
        del _pending[:len(batch)]
        lib = _native.lib()
        n = len(batch)
        descs = (_GemmDesc * n)()
        for i, (a2, b2, out, M, N, K, acc, _done) in enumerate(batch):
            descs[i] = _GemmDesc(a2.data_ptr(), b2.data_ptr(), out.data_ptr(), M, N, K, a2.stride(0), b2.stride(0),
                                 out.stride(0), int(out.dtype == torch.float32), int(acc))
        if not _TAIL_SPLIT:
            lib.zen_gemm2_tail_split(0)
        ws, n_ws, cnt, n_cnt = _workspace_args(batch[0][0].device) if _TAIL_SPLIT else (0, 0, 0, 0)
        rc = lib.zen_gemm_bf16_2cta_group(descs, n, 1, 1, ws, n_ws, cnt, n_cnt, _native.stream_ptr())
        _native.check(rc, "zen_gemm_bf16_2cta_group")
        for item in batch:
            if item[7] is not None:
                item[7]()
    from . import elementwise as _E

    _E.flush_colreduce()                           # the bias / norm-parameter reductions queued beside them


def _finish(r, bias, out, accumulate, dtype):
    if bias is not None:
        r = r + bias.float()
    if out is not None:
        if accumulate:
            out.add_(r.to(out.dtype))
        else:
            out.copy_(r.to(out.dtype))
        return out
    return r.to(dtype)


def gemm_error() -> int:
    """Error code of the last tcgen05 kernel that gave up a bounded wait (0 = none)."""
    lib = _native.lib()
    return int(lib.zen_gemm_error()) or int(lib.zen_gemm2_error()) or int(lib.zen_gemm_splitk_error())

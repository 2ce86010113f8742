"""Kernel entry points on torch CUDA tensors.

Each function hands its tensors to the native binding (``csrc/host/torch_ops.cpp``), which validates
shapes, prepares operands, allocates outputs and calls ``libghost_b200.so`` on torch's current
stream; a few rarely called ones do so here through ctypes.  The arithmetic runs in the library's
kernels.  Scratch memory comes from a grow-only arena per (device, stream), so no allocation happens
in steady state and nothing is freed while kernels that use it may still be queued.
"""
from __future__ import annotations

from typing import Dict, Optional, Tuple

import torch

from . import _lib

_BF16 = torch.bfloat16
_F32 = torch.float32

_native = _lib.native


class _Arenas:
    """The native binding's workspaces."""

    @staticmethod
    def clear() -> None:
        """Give every workspace back to torch's allocator."""
        _native().arena_clear()


_arenas = _Arenas()

_timing: Optional[list] = None


def start_kernel_timing() -> None:
    """Bracket every library call with CUDA events on the launching stream (opt-in; used by the
    benchmark to attribute device time and algorithmic work to kernel groups)."""
    global _timing
    _timing = []


def stop_kernel_timing() -> dict:
    """Synchronise and return ``{'ops': {name: {calls, ms, flops, bytes, bound}}, 'share': {...}}``."""
    global _timing
    records, _timing = _timing or [], None
    torch.cuda.synchronize()
    out: Dict[str, dict] = {}
    for name, bound, flops, nbytes, e0, e1 in records:
        r = out.setdefault(name, {"calls": 0, "ms": 0.0, "flops": 0.0, "bytes": 0.0, "bound": bound})
        r["calls"] += 1
        r["ms"] += e0.elapsed_time(e1)
        r["flops"] += flops
        r["bytes"] += nbytes
    total = sum(r["ms"] for r in out.values()) or 1.0
    return {"ops": out, "share": {k: round(v["ms"] / total, 4) for k, v in out.items()},
            "total_ms": total}


class _Timed:
    """``with _Timed(name, bound, flops, bytes):`` around the library calls of one op."""

    def __init__(self, name: str, bound: str, flops: float, nbytes: float):
        self.rec = (name, bound, float(flops), float(nbytes))

    def __enter__(self):
        if _timing is not None:
            self.e0 = torch.cuda.Event(enable_timing=True)
            self.e0.record()
        return self

    def __exit__(self, *exc):
        if _timing is not None and exc[0] is None:
            e1 = torch.cuda.Event(enable_timing=True)
            e1.record()
            _timing.append(self.rec + (self.e0, e1))
        return False


def _stream_ptr() -> int:
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def _require_cuda(*tensors: torch.Tensor) -> None:
    for t in tensors:
        if not t.is_cuda:
            raise RuntimeError("ghostsuite_b200 kernels need CUDA tensors (no CPU fallback exists)")


def _dt_flag(t: torch.Tensor) -> int:
    if t.dtype == _F32:
        return 1
    if t.dtype == _BF16:
        return 0
    raise ValueError(f"unsupported dtype {t.dtype}: the kernels take float32 or bfloat16")


def _as3d(x: torch.Tensor) -> torch.Tensor:
    """[N, d] -> [N, 1, d]; [N, ..., d] -> [N, T, d] (contiguous).  float16 / float64 inputs are
    widened / narrowed to float32 first (the kernels take float32 and bfloat16)."""
    if x.dtype in (torch.float16, torch.float64):
        x = x.float()
    if x.dim() <= 2:
        x = x.unsqueeze(1)
    else:
        x = x.reshape(x.shape[0], -1, x.shape[-1])
    return x.contiguous()


def _tma_ready(x: torch.Tensor) -> bool:
    return x.dtype == _BF16 and x.shape[-1] % 8 == 0 and x.data_ptr() % 16 == 0


def _pad8(n: int) -> int:
    return (n + 7) // 8 * 8


def _cast(lib, src: torch.Tensor, samples: int, T: int, dst_ptr: int, ld_dst: int, cpad: int,
          kinds: Tuple[int, ...], row_stack: bool) -> None:
    k = tuple(kinds) + (0,) * (3 - len(kinds))
    _lib.check(lib.ghost_cast_split_bf16(src.data_ptr(), _dt_flag(src), samples, T, src.shape[-1],
                                         src.shape[-1], dst_ptr, ld_dst, cpad, len(kinds),
                                         k[0], k[1], k[2], 1 if row_stack else 0, _stream_ptr()))


#: hi/lo layout of the projection matrices of an fp32 model, the right operand of
#: ``sum_k L[k] R[k] = hi*hi + lo*hi + hi*lo``
_SPLIT_RIGHT = (0, 0, 1)


def _cols(x: torch.Tensor) -> int:
    return int(x.shape[-1])


def _rows(x: torch.Tensor) -> int:
    return x.numel() // max(1, int(x.shape[-1]))


# --------------------------------------------------------------------------------------------
# Linear / Conv1D weight dot product: Gram path
# --------------------------------------------------------------------------------------------
def gram_dot(A: torch.Tensor, G: torch.Tensor, n_val: int, round_mode: int = 0,
             scale: float = 1.0) -> torch.Tensor:
    """Full ``[n_val, n_train]`` dot-product matrix through the fused Gram kernel.

    bf16 inputs are used as they are (copied only if their feature size is not a multiple of 8);
    fp32 inputs are split into bf16 hi/lo parts so the result keeps fp32-class accuracy.
    """
    if _timing is None:
        return _native().gram_dot(A, G, n_val, round_mode, scale)
    # algorithmic work (the fp32 hi/lo split executes three times this on the tensor pipe)
    N, T = A.shape[0], max(1, _rows(A) // A.shape[0])
    width = _cols(A) + _cols(G)
    with _Timed("ghost_gram_kernel", "tensor", 2.0 * (N - n_val) * T * n_val * T * width,
                float(A.element_size()) * N * T * width):
        return _native().gram_dot(A, G, n_val, round_mode, scale)


# --------------------------------------------------------------------------------------------
# train-gradient recovery and the per-sample-gradient path
# --------------------------------------------------------------------------------------------
def wgrad(X: torch.Tensor, Y: torch.Tensor, scale: float, out_dtype: torch.dtype,
          out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
    """``scale * sum over all rows of X^T Y`` -> ``[X.shape[-1], Y.shape[-1]]`` in ``out_dtype``.

    ``X``/``Y`` are ``[samples, T, cols]`` (train samples only).
    """
    if out is None and out_dtype not in (_F32, _BF16):
        raise ValueError(f"unsupported dtype {out_dtype}: the kernels take float32 and bfloat16")
    if _timing is None:
        return _native().wgrad(X, Y, scale, out_dtype is _F32, out, accumulate)
    with _Timed("xty_gemm_pair_kernel[wgrad]", "tensor", 2.0 * _rows(X) * _cols(X) * _cols(Y),
                2.0 * _rows(X) * (_cols(X) + _cols(Y))):
        return _native().wgrad(X, Y, scale, out_dtype is _F32, out, accumulate)


_PERSAMPLE_NAME = "xty_gemm_pair_kernel+tile_dot_mma_kernel[persample]"


_COLSUM_FLAG = {None: 0, "X": 1, "Y": 2}


def persample_dot(X: torch.Tensor, Y: torch.Tensor, n_val: int, dot_scale: float = 1.0,
                  want_grad: bool = False, grad_scale: float = 1.0,
                  grad_dtype: Optional[torch.dtype] = None, colsum_of: Optional[str] = None):
    """Dot-product matrix through explicit per-sample weight gradients kept in tensor memory.

    ``X``/``Y``: ``[N, T, cols]``, train first.  Returns ``(M[n_val, n_train], train_grad or None)``
    with ``train_grad = grad_scale * sum_b X_b^T Y_b`` of shape ``[X cols, Y cols]``.  With
    ``colsum_of='X'`` or ``'Y'`` a third value is returned: the per-sample column sums ``[N, cols]``
    (float32) of that operand, taken inside the GEMM pass, or None when the operands are fp32 (their
    bf16 hi/lo split is what the kernel sees).
    """
    if colsum_of not in _COLSUM_FLAG:
        raise ValueError("colsum_of must be None, 'X' or 'Y'")
    gdt = grad_dtype if grad_dtype is not None else (_BF16 if X.dtype is _BF16 else _F32)
    if want_grad and gdt is not _F32 and gdt is not _BF16:
        raise ValueError(f"unsupported dtype {gdt}: the kernels take float32 and bfloat16")
    args = (X, Y, n_val, dot_scale, want_grad, grad_scale, gdt is _F32, _COLSUM_FLAG[colsum_of])
    if _timing is None:
        res = _native().persample_dot(*args)
    else:
        m, n, rows, N = _cols(X), _cols(Y), _rows(X), X.shape[0]
        with _Timed(_PERSAMPLE_NAME, "tensor", 2.0 * rows * m * n + 2.0 * n_val * (N - n_val) * m * n,
                    2.0 * rows * (m + n)):
            res = _native().persample_dot(*args)
    return res if colsum_of is not None else res[:2]


def _dtype_code(dt: Optional[torch.dtype]) -> int:
    return -1 if dt is None else (1 if dt is _F32 else 0)


def dense_hook(A: torch.Tensor, B: torch.Tensor, n_val: int, weight_is_in_by_out: bool, use_gram: bool,
               grad_dtype: Optional[torch.dtype], grad_scale: float, has_bias: bool,
               bias_grad_dtype: Optional[torch.dtype], any_path: bool = True, fuse_colsums: bool = True):
    """All that the backward hook of a Linear / Conv1D layer needs, in one native call: ``(M, weight
    gradient, column sums of B, bias matrix, bias gradient)``, None where not wanted (a dtype of None,
    no bias).  With ``any_path`` a layer of few token rows takes the one-launch kernel of
    ``ghost_dense_small`` whatever ``use_gram`` says.  Without ``fuse_colsums`` the column sums take a launch of
    their own instead of falling out of another kernel's pass over ``B``.  The last two are allocated
    only: they are filled by the launch that ends the backward pass (:func:`pass_reduce`)."""
    args = (A, B, n_val, weight_is_in_by_out, use_gram, _dtype_code(grad_dtype), grad_scale, has_bias,
            _dtype_code(bias_grad_dtype), any_path, fuse_colsums)
    if _timing is None:
        return _native().dense_hook(*args)
    d, p, rows, N = _cols(A), _cols(B), _rows(A), A.shape[0]
    if use_gram:
        T = rows // N
        name, flops = "ghost_gram_kernel+xty_gemm_pair_kernel", 2.0 * (N - n_val) * T * (n_val * T * (d + p) + d * p)
    else:
        name, flops = _PERSAMPLE_NAME, 2.0 * rows * d * p + 2.0 * n_val * (N - n_val) * d * p
    with _Timed(name, "tensor", flops, 2.0 * rows * (d + p)):
        return _native().dense_hook(*args)


def conv_hook(A: torch.Tensor, B: torch.Tensor, n_val: int, window: Tuple[int, ...], use_gram: bool,
              grad_dtype: Optional[torch.dtype], grad_scale: float, has_bias: bool,
              bias_grad_dtype: Optional[torch.dtype]):
    """:func:`dense_hook` for a Conv2d (groups == 1): ``A [N, C, H, W]``, ``B [N, p, Ho, Wo]``, ``window =
    (kh, kw, stride y, x, padding y, x, dilation y, x)``.  Output positions are the tokens; the operands are
    laid out for the tensor-core paths straight from these tensors.  The weight gradient is ``[p, C*kh*kw]``."""
    args = (A, B, n_val, window, use_gram, _dtype_code(grad_dtype), grad_scale, has_bias, _dtype_code(bias_grad_dtype))
    if _timing is None:
        return _native().conv_hook(*args)
    N, p, T, d = A.shape[0], B.shape[1], B.shape[2] * B.shape[3], A.shape[1] * window[0] * window[1]
    with _Timed(_PERSAMPLE_NAME, "tensor", 2.0 * N * T * d * p + 2.0 * n_val * (N - n_val) * d * p, 2.0 * N * T * (d + p)):
        return _native().conv_hook(*args)


def persample_tiles(X: torch.Tensor, Y: torch.Tensor, sample0: int, samples: int,
                    colsum_of: Optional[str] = None, colsums: Optional[torch.Tensor] = None) -> torch.Tensor:
    """First pass of the per-sample path alone: the bf16 tiles ``X_s^T Y_s`` of samples
    ``[sample0, sample0 + samples)``, laid out ``[tiles, samples, 32768]`` (128 x 256 tiles).  ``X`` /
    ``Y``: contiguous bf16 ``[N, T, cols]`` with column counts that are multiples of 8.  With
    ``colsum_of`` the rows ``sample0 ..`` of ``colsums`` (``[N, cols]`` float32) are filled too."""
    lib = _lib.load()
    N, T, m = X.shape
    n = Y.shape[-1]
    nbytes = int(lib.ghost_persample_tiles_bytes(samples, m, n))
    tiles = torch.empty((nbytes // (samples * 65536), samples, 32768), dtype=_BF16, device=X.device)
    cs_flag = 0 if colsum_of is None else (1 if colsum_of == "X" else 2)
    with _Timed(_PERSAMPLE_NAME, "tensor", 2.0 * samples * T * m * n, 2.0 * samples * T * (m + n)):
        _lib.check(lib.ghost_persample_tiles_bf16(
            X.data_ptr(), Y.data_ptr(), N, T, m, n, m, n, int(sample0), int(samples), cs_flag,
            colsums.data_ptr() if cs_flag else None, tiles.data_ptr(), nbytes, _stream_ptr()))
    return tiles


def tile_dot(V: torch.Tensor, W: torch.Tensor, m: int, n: int, dot_scale: float = 1.0,
             want_grad: bool = False, grad_scale: float = 1.0, grad_dtype: torch.dtype = _BF16,
             M: Optional[torch.Tensor] = None, grad: Optional[torch.Tensor] = None):
    """Second pass alone.  ``W``: train tiles ``[tiles, n_train, 32768]``; ``V``: validation tiles, either
    ``[tiles, n_val, 32768]`` or, as an all-gather over ranks leaves them, ``[ranks, tiles, per_rank,
    32768]`` (validation sample ``r * per_rank + i`` of the result is sample ``i`` of rank ``r``).
    Returns ``(M[n_val, n_train], train_grad[m, n] or None)``, written into ``M`` / ``grad`` when given."""
    lib = _lib.load()
    if V.dim() == 3:
        V = V.unsqueeze(0)
    ranks, tiles, per_rank, _ = V.shape
    n_train = W.shape[1]
    n_val = ranks * per_rank
    if M is None:
        M = torch.empty((n_val, n_train), dtype=_F32, device=W.device)
    if want_grad and grad is None:
        grad = torch.empty((m, n), dtype=grad_dtype, device=W.device)
    with _Timed(_PERSAMPLE_NAME, "tensor", 2.0 * n_val * n_train * m * n, 0.0):
        _lib.check(lib.ghost_tile_dot_bf16(
            V.data_ptr(), ranks, per_rank, W.data_ptr(), n_train, m, n, float(dot_scale), M.data_ptr(),
            grad.data_ptr() if want_grad else None, _dt_flag(grad) if want_grad else 0, float(grad_scale), 0,
            _stream_ptr()))
    return M, (grad if want_grad else None)


# Streaming passes that wait for an all-gather in flight, per (device, stream): the pass of one layer
# is launched when the next layer has launched its own tile passes and all-gather (or by
# ``finish_exchange_jobs``), so the transfer runs under that layer's GEMMs.
_exchange_jobs: Dict[Tuple[int, int], list] = {}

#: how many layers' streaming passes may wait for their all-gather at a time (each holds its tile
#: buffers); a pass is launched when this many later layers have issued theirs
EXCHANGE_DEPTH = 1


def _finish_exchange_job(job: dict) -> None:
    job["work"].wait()               # the current stream waits for the all-gather
    tile_dot(job["V"], job["W"], job["m"], job["n"], job["dot_scale"], job["grad"] is not None,
             job["grad_scale"], _BF16, M=job["M"], grad=job["grad"])
    cb = job["on_ready"]
    job.clear()
    if cb is not None:
        cb()


def finish_exchange_jobs() -> None:
    """Launch the streaming pass of every layer that still waits for its all-gather."""
    if not _exchange_jobs:
        return
    for key in list(_exchange_jobs):
        for job in _exchange_jobs.pop(key):
            _finish_exchange_job(job)


def persample_dot_exchanged(X: torch.Tensor, Y: torch.Tensor, n_val_local: int, exchange, dot_scale: float = 1.0,
                            want_grad: bool = False, grad_scale: float = 1.0,
                            grad_dtype: Optional[torch.dtype] = None, colsum_of: Optional[str] = None,
                            on_ready=None):
    """The per-sample path of a rank that holds ``n_val_local`` of the validation samples (the last
    rows of ``X`` / ``Y``): tiles of the local validation samples, an all-gather of them along
    dimension 0 over ``exchange.world`` ranks (``exchange.gather_rows``), tiles of the local train
    samples, then the contraction of ALL validation tiles with the local train tiles.  Returns
    ``(M[world * n_val_local, n_train], train_grad or None, colsums of the LOCAL samples or None)``, or
    None when the shapes are outside what the two-pass entry points take (fp32 operands, a bf16
    train gradient of more than 32 samples, a validation split that does not fit the kernel's row
    blocks).

    With ``on_ready`` and an exchange that has ``gather_rows_async`` the all-gather is not waited
    for: ``M`` and the gradient are filled by a later launch -- when the next call on this stream has
    enqueued its own tile passes, or in :func:`finish_exchange_jobs` -- and ``on_ready()`` is called
    right after that launch has been enqueued."""
    _require_cuda(X, Y)
    if X.dtype != _BF16 or Y.dtype != _BF16:
        return None
    X, Y = _as3d(X), _as3d(Y)
    N, T, m = X.shape
    n = Y.shape[-1]
    n_train = N - n_val_local
    ranks = int(exchange.world)
    if n_train <= 0:
        raise ValueError("No training samples to compute dot product, check batch sizes.")
    if n_val_local <= 0 or Y.shape[0] != N or Y.shape[1] != T or not (_tma_ready(X) and _tma_ready(Y)):
        return None
    gdt = grad_dtype or X.dtype
    if want_grad and gdt != _F32 and n_train > 32:
        return None
    n_val = n_val_local * ranks
    block = 8 if n_val <= 8 else (16 if n_val <= 16 else 32)
    if block % n_val_local != 0 and n_val_local % block != 0:
        return None
    if colsum_of not in (None, "X", "Y"):
        raise ValueError("colsum_of must be None, 'X' or 'Y'")
    colsums = None
    if colsum_of is not None:
        colsums = torch.empty((N, m if colsum_of == "X" else n), dtype=_F32, device=X.device)
    V_loc = persample_tiles(X, Y, n_train, n_val_local, colsum_of, colsums)
    deferred = on_ready is not None and hasattr(exchange, "gather_rows_async")
    if deferred:
        V_all, work = exchange.gather_rows_async(V_loc.unsqueeze(0))
    else:
        V_all = exchange.gather_rows(V_loc.unsqueeze(0))     # [ranks, tiles, n_val_local, 32768]
    W = persample_tiles(X, Y, 0, n_train, colsum_of, colsums)
    if not deferred:
        M, grad = tile_dot(V_all, W, m, n, dot_scale, want_grad, grad_scale, gdt)
        return M, grad, colsums
    M = torch.empty((n_val, n_train), dtype=_F32, device=X.device)
    grad = torch.empty((m, n), dtype=gdt, device=X.device) if want_grad else None
    key = (X.device.index if X.device.index is not None else torch.cuda.current_device(), _stream_ptr())
    queue = _exchange_jobs.setdefault(key, [])
    queue.append({"V": V_all, "W": W, "work": work, "m": m, "n": n, "dot_scale": dot_scale,
                  "grad_scale": grad_scale, "M": M, "grad": grad, "on_ready": on_ready})
    while len(queue) > max(1, int(EXCHANGE_DEPTH)):
        _finish_exchange_job(queue.pop(0))
    return M, grad, colsums


# --------------------------------------------------------------------------------------------
# bias / LayerNorm / small reductions
# --------------------------------------------------------------------------------------------
def colsum(G: torch.Tensor) -> torch.Tensor:
    """Per-sample column sums over tokens: ``[N, T, p] -> [N, p]`` float32."""
    if _timing is None:
        return _native().colsum(G)
    with _Timed("colsum_kernel", "hbm", 0.0, float(G.numel()) * G.element_size()):
        return _native().colsum(G)


def small_gram(X: torch.Tensor, n_val: int, scale: float = 1.0) -> torch.Tensor:
    """``M[v, b] = scale * <X[n_train + v], X[b]>`` for per-sample float32 vectors ``X[N, F]``."""
    lib = _lib.load()
    _require_cuda(X)
    if X.dtype != _F32 or X.dim() != 2 or not X.is_contiguous():
        raise ValueError("small_gram takes a contiguous float32 [N, F] tensor")
    n_train = X.shape[0] - n_val
    if n_train <= 0:
        raise ValueError("No training samples to compute dot product, check batch sizes.")
    M = torch.empty((n_val, n_train), dtype=_F32, device=X.device)
    with _Timed("small_gram_kernel", "hbm", 0.0, 4.0 * X.numel()):
        _lib.check(lib.ghost_small_gram_f32(X.data_ptr(), n_train, n_val, X.shape[1], float(scale),
                                            M.data_ptr(), _stream_ptr()))
    return M


def rows_sum(X: torch.Tensor, n_rows: int, scale: float, out_dtype: torch.dtype,
             out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
    """``scale * X[:n_rows].sum(0)`` cast to ``out_dtype`` (optionally accumulated into ``out``)."""
    lib = _lib.load()
    _require_cuda(X)
    if X.dtype != _F32 or X.dim() != 2 or not X.is_contiguous():
        raise ValueError("rows_sum takes a contiguous float32 [N, F] tensor")
    if out is None:
        out = torch.empty((X.shape[1],), dtype=out_dtype, device=X.device)
        accumulate = False
    with _Timed("rows_sum_kernel", "hbm", 0.0, 4.0 * n_rows * X.shape[1]):
        _lib.check(lib.ghost_rows_sum(X.data_ptr(), int(n_rows), X.shape[1], float(scale), out.data_ptr(),
                                      _dt_flag(out), 1 if accumulate else 0, _stream_ptr()))
    return out


def small_reduce_batch(jobs) -> None:
    """Run many :func:`small_gram` / :func:`rows_sum` reductions in one launch per 48 of them.
    ``jobs``: dicts with ``X`` (contiguous float32 ``[n_train + n_val, F]``), ``n_train``, ``n_val`` and
    optionally ``M`` (float32 ``[n_val, n_train]`` output, with ``dot_scale``) and ``sum_out``
    (float32 / bfloat16 ``[F]`` output, with ``sum_scale``); the outputs are written in place.  A job
    with ``Xv = (gathered, offset, per_rank)`` takes its validation rows from ``gathered[r, offset + i
    * F : ...]`` (row ``r * per_rank + i``; ``gathered`` is a contiguous float32 ``[ranks, pitch]`` tensor, the
    result of one all-gather that carried many jobs' validation rows) and only its train rows from
    ``X``."""
    jobs = list(jobs)
    for first in range(0, len(jobs), 48):
        pass_reduce(jobs[first:first + 48], [])


def pass_reduce(jobs: list, matrices: list) -> list:
    """What is left to reduce when a backward pass ends, in one launch: the jobs of
    :func:`small_reduce_batch`, and for every ``[n_val, n_train]`` float32 matrix its sum over the
    validation samples (returned as a list of ``[n_train]`` tensors; a matrix may be one that a job
    of the same call fills)."""
    if _timing is None:
        return _native().pass_reduce(jobs, matrices)
    with _Timed("pass_reduce_kernel", "hbm", 0.0, 4.0 * sum(j["X"].numel() for j in jobs)):
        return _native().pass_reduce(jobs, matrices)


def finish_pass(jobs: list, dots: list, observer) -> bool:
    """:func:`pass_reduce` for the lists that the hooks fill, and what follows it, in one native call: every
    ``(parameter, matrix)`` of ``dots`` -- a parameter's last one counts -- gets its vector as
    ``parameter.grad_dot_prod``, if ``grad_dot_prod_matrix`` still is that matrix, and the train gradient of every
    job with a ``param`` becomes ``param.train_grad`` or is added to it, whereupon ``observer(param)`` is called.
    False, with nothing done, when a matrix is not on a GPU or the library calls are timed one by one."""
    if _timing is not None or (dots and not dots[0][1].is_cuda) or not _lib.binding_present():
        return False
    return _native().finish_pass(jobs, dots, observer)


def matrix_sum(matrices: list) -> torch.Tensor:
    """Sum of equal ``[n_val, n_train]`` float32 matrices as one flat float32 buffer: the matrix, its
    column sums (``n_train`` values), and the device error word (the bits of an int32)."""
    if _timing is None:
        return _native().matrix_sum(matrices)
    with _Timed("matrix_sum_kernel", "hbm", 0.0, 4.0 * len(matrices) * matrices[0].numel()):
        return _native().matrix_sum(matrices)


def layernorm_persample(A: torch.Tensor, G: torch.Tensor, eps: float, rms: bool = False
                        ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per-sample LayerNorm gamma/beta gradients ``([N, F], [N, F])`` float32 in one pass.  With
    ``rms=True`` the normalisation is RMS norm's (no centring); the second result is then just the
    token sum of the out-grad."""
    if _timing is None:
        return _native().norm_persample(A, G, eps, rms)
    with _Timed("layernorm_persample_kernel", "hbm", 0.0, 2.0 * A.numel() * A.element_size() + 8.0 * A.shape[0] * _cols(A)):
        return _native().norm_persample(A, G, eps, rms)


def norm_hook(A: torch.Tensor, G: torch.Tensor, eps: float, rms: bool, n_val: int, weight_dtype: torch.dtype,
              bias_dtype: Optional[torch.dtype]):
    """:func:`layernorm_persample` plus what the launch that ends the backward pass fills:
    ``(gw, gb, weight matrix, bias matrix, weight gradient, bias gradient)``; no bias: a dtype of None."""
    args = (A, G, eps, rms, n_val, _dtype_code(weight_dtype), _dtype_code(bias_dtype))
    if _timing is None:
        return _native().norm_hook(*args)
    with _Timed("layernorm_persample_kernel", "hbm", 0.0, 2.0 * A.numel() * A.element_size() + 8.0 * A.shape[0] * _cols(A)):
        return _native().norm_hook(*args)


# --------------------------------------------------------------------------------------------
# Embedding
# --------------------------------------------------------------------------------------------
def embedding_dot(ids: torch.Tensor, G: torch.Tensor, n_val: int, vocab: int,
                  scale: float = 1.0) -> torch.Tensor:
    if _timing is None:
        return _native().embedding_dot(ids, G, n_val, vocab, scale)
    with _Timed("emb_dot_kernel", "hbm", 0.0, float(G.numel()) * G.element_size() + 8.0 * ids.numel()):
        return _native().embedding_dot(ids, G, n_val, vocab, scale)


def embedding_wgrad(ids: torch.Tensor, G: torch.Tensor, n_train: int, vocab: int, pre_scale: float,
                    divisor: float, out: Optional[torch.Tensor] = None,
                    accumulate: bool = False) -> torch.Tensor:
    """Averaged train gradient of an embedding table ``[vocab, d]`` in the dtype of ``G``."""
    args = (ids, G, n_train, vocab, pre_scale, divisor, out, accumulate)
    if _timing is None:
        return _native().embedding_wgrad(*args)
    share = n_train / max(1, G.shape[0])
    with _Timed("emb_grad_kernel", "hbm", 0.0,
                (share * G.numel() + float(vocab) * _cols(G)) * G.element_size() + 8.0 * share * ids.numel()):
        return _native().embedding_wgrad(*args)


def embedding_hook(ids: torch.Tensor, G: torch.Tensor, n_val: int, vocab: int, pre_scale: float):
    """:func:`embedding_dot` and :func:`embedding_wgrad` (divided by the train samples) from one set of
    buckets: ``(M[n_val, n_train], train gradient [vocab, d] in the dtype of G)``."""
    args = (ids, G, n_val, vocab, pre_scale)
    if _timing is None:
        return _native().embedding_hook(*args)
    with _Timed("emb_join_kernel+emb_grad_kernel", "hbm", 0.0,
                (float(G.numel()) + float(vocab) * _cols(G)) * G.element_size() + 8.0 * ids.numel()):
        return _native().embedding_hook(*args)


# --------------------------------------------------------------------------------------------
# GradProj
# --------------------------------------------------------------------------------------------
def prepare_projection(P: torch.Tensor, split: bool) -> torch.Tensor:
    """bf16 copy of a projection matrix ``[k, n]`` laid out for the kernel: columns padded to a
    multiple of 8; for fp32 models the hi/lo split matching ``_SPLIT_RIGHT``."""
    lib = _lib.load()
    _require_cuda(P)
    P = P.contiguous()
    k, n = P.shape
    cp = _pad8(n)
    parts = _SPLIT_RIGHT if split else (0,)
    out = torch.empty((k, len(parts) * cp), dtype=_BF16, device=P.device)
    _cast(lib, P, 1, k, out.data_ptr(), len(parts) * cp, cp, parts, False)
    return out


def gradproj_dense(G: torch.Tensor, A: torch.Tensor, P_r: torch.Tensor, P_c: torch.Tensor,
                   k_r: int, k_c: int, scale: float, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[b] = scale * (G_b P_r^T)^T (A_b P_c^T)`` written into ``out`` (``[B, >= k_r*k_c]`` fp32,
    possibly a column slice of a wider row-major buffer), or into a new ``[B, k_r, k_c]`` tensor.  ``P_r``/``P_c`` come from
    :func:`prepare_projection` (split layout iff the activations are fp32)."""
    if _timing is None:
        return _native().gradproj_dense(G, A, P_r, P_c, k_r, k_c, scale, out)
    n_r, n_c = _cols(G), _cols(A)
    with _Timed("gradproj_kernel", "hbm", 2.0 * _rows(G) * (n_r * k_r + n_c * k_c + k_r * k_c),
                float(_rows(G)) * (n_r + n_c) * G.element_size() + 2.0 * (k_r * n_r + k_c * n_c)
                + 4.0 * G.shape[0] * k_r * k_c):
        return _native().gradproj_dense(G, A, P_r, P_c, k_r, k_c, scale, out)


def prepare_embedding_projection(P_i: torch.Tensor) -> torch.Tensor:
    """``P_i [k_i, vocab]`` as the embedding-projection kernel reads it: float32 ``[vocab, k_i]``, so
    that a token id selects one contiguous row (made once per layer)."""
    _require_cuda(P_i)
    return P_i.detach().to(_F32).t().contiguous()


def gradproj_embedding(ids: torch.Tensor, G: torch.Tensor, P_o_prepared: torch.Tensor, P_i_t: torch.Tensor,
                       k_o: int, k_i: int, scale: float = 1.0,
                       out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[b] = scale * sum_t (P_o g_bt)(P_i[:, id_bt])^T`` as ``[B, k_o*k_i]`` float32 (written into
    ``out`` when given: a ``[B, >= k_o*k_i]`` row-major view, e.g. a column slice of the engine's
    buffer).  ``P_o_prepared`` comes from :func:`prepare_projection` (split layout iff ``G`` is
    float32), ``P_i_t`` from :func:`prepare_embedding_projection`."""
    if _timing is None:
        return _native().gradproj_embedding(ids, G, P_o_prepared, P_i_t, k_o, k_i, scale, out)
    rows, d = ids.numel(), _cols(G)
    with _Timed("gradproj_kernel", "hbm", 2.0 * rows * (d * k_o + k_o * k_i),
                float(rows) * (d * G.element_size() + 8 + 4 * k_i) + 4.0 * ids.shape[0] * k_o * k_i):
        return _native().gradproj_embedding(ids, G, P_o_prepared, P_i_t, k_o, k_i, scale, out)


#: largest block (rows of either operand) the similarity kernel is used for whatever the rows' type.  Beyond it a
#: library GEMM takes float32 rows more accurately (192 x 192 scores over 98304 elements of both signs: 1.2e-6 off the
#: 64-bit result against 4.4e-6; 494 us against 97); bfloat16 rows: projection_utils._bf16_sets_for_kernel
SIMILARITY_KERNEL_MAX_ROWS = 128


def projection_similarity(P1: torch.Tensor, P2: torch.Tensor, scale: float = 1.0) -> torch.Tensor:
    """``scale * P1 @ P2.T`` -> ``[n1, n2]`` float32 for two blocks of projection rows (float32 or
    bfloat16, same dtype, unit stride along the projection dimension)."""
    if _timing is None:
        return _native().projection_similarity(P1, P2, scale)
    with _Timed("proj_similarity_kernel", "hbm", 2.0 * P1.shape[0] * P2.numel(),
                float(P1.numel() + P2.numel()) * P1.element_size()):
        return _native().projection_similarity(P1, P2, scale)


def launch_count() -> int:
    return _lib.launch_count()


# ------------------------------------------------------------------------------------------------
# benchmark model helper: fused token cross-entropy (not part of the ghost hot path)
# ------------------------------------------------------------------------------------------------
def ce_supported(logits: torch.Tensor) -> bool:
    """True when the fused loss kernels can take this [rows, cols] logit matrix as it is."""
    if not logits.is_cuda or logits.dtype not in (_BF16, _F32) or logits.dim() != 2:
        return False
    vec = 8 if logits.dtype == _BF16 else 4
    return logits.stride(1) == 1 and logits.stride(0) % vec == 0 and logits.data_ptr() % 16 == 0


def ce_forward(logits: torch.Tensor, targets: torch.Tensor, valid_cols: int, ignore_index: int = -100,
               grad_scale: Optional[torch.Tensor] = None):
    """Per-row log-sum-exp over the first ``valid_cols`` columns and per-row loss (0 for ignored
    rows), both float32 ``[rows]``, in one pass over ``logits``.  With ``grad_scale`` (one-element
    float32 device tensor) the kernel also writes ``grad_scale * (softmax - onehot)`` in the logits'
    dtype and returns it as a third value."""
    lib = _lib.load()
    _require_cuda(logits, targets)
    rows, cols = logits.shape
    targets = targets.contiguous()
    lse = torch.empty(rows, dtype=_F32, device=logits.device)
    loss_rows = torch.empty(rows, dtype=_F32, device=logits.device)
    dlogits = torch.empty((rows, cols), dtype=logits.dtype, device=logits.device) if grad_scale is not None else None
    nbytes = float(rows) * valid_cols * logits.element_size() * (1.0 if dlogits is None else 2.0)
    with _Timed("ce_forward_kernel", "hbm", 0.0, nbytes):
        _lib.check(lib.ghost_workload_ce_forward(logits.data_ptr(), _dt_flag(logits), rows, cols, int(valid_cols),
                                                 logits.stride(0), targets.data_ptr(), int(ignore_index),
                                                 lse.data_ptr(), loss_rows.data_ptr(),
                                                 grad_scale.data_ptr() if grad_scale is not None else None,
                                                 dlogits.data_ptr() if dlogits is not None else None,
                                                 _stream_ptr()))
    if grad_scale is None:
        return lse, loss_rows
    return lse, loss_rows, dlogits


def ce_rescale_(dlogits: torch.Tensor, upstream: torch.Tensor) -> torch.Tensor:
    """``dlogits *= upstream[0]`` in place; the kernel returns at once when the factor is exactly 1."""
    lib = _lib.load()
    _require_cuda(dlogits, upstream)
    rows, cols = dlogits.shape
    with _Timed("ce_rescale_kernel", "hbm", 0.0, 0.0):
        _lib.check(lib.ghost_workload_ce_rescale(dlogits.data_ptr(), _dt_flag(dlogits), rows, cols,
                                                 upstream.data_ptr(), _stream_ptr()))
    return dlogits


def ce_backward(logits: torch.Tensor, targets: torch.Tensor, valid_cols: int, lse: torch.Tensor,
                scale: torch.Tensor, ignore_index: int = -100) -> torch.Tensor:
    """``scale * (softmax(logits[:, :valid_cols]) - onehot(targets))`` in the logits' dtype, zero in
    padded columns and ignored rows; ``scale`` is a one-element float32 device tensor."""
    lib = _lib.load()
    _require_cuda(logits, targets, lse, scale)
    rows, cols = logits.shape
    targets = targets.contiguous()
    out = torch.empty((rows, cols), dtype=logits.dtype, device=logits.device)
    with _Timed("ce_backward_kernel", "hbm", 0.0, 2.0 * rows * cols * logits.element_size()):
        _lib.check(lib.ghost_workload_ce_backward(logits.data_ptr(), _dt_flag(logits), rows, cols, int(valid_cols),
                                                  logits.stride(0), targets.data_ptr(), int(ignore_index),
                                                  lse.data_ptr(), scale.data_ptr(), out.data_ptr(), cols,
                                                  _stream_ptr()))
    return out

"""Projection-rank selection and projection-matrix initialisers for GradProj.

Drop-in for GhostSuite's ``ghostEngines/gradProjection/projection_utils.py``: ``choose_ki_ko``
(:12-66), the Gaussian / Rademacher / row-orthonormal initialisers (:69-174) and
``compute_projection_metadata`` (:202-238) return the same values for the same arguments, so that a
projection matrix built here equals the one the reference builds from the same seed on the same
device type.  This is one-time setup and stays in PyTorch.
"""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch
import torch.nn as nn

from ... import ops


def choose_ki_ko(n_i: int, n_o: int, k_total: int, k_min: int = 1) -> Tuple[int, int]:
    """Pick ``(k_i, k_o)`` with ``k_i * k_o ~ k_total``, ``k_i / k_o ~ sqrt(n_o / n_i)`` and both at
    least ``k_min`` (and at most the layer dimension), then search the +-2 neighbourhood for the
    product closest to ``k_total``; the first best candidate in row-major (di, dj) order wins."""
    if min(n_i, n_o) <= 0 or k_total <= 0:
        raise ValueError(f"Invalid dimensions for projection: n_i={n_i}, n_o={n_o}, k_total={k_total}")
    if k_min > min(n_i, n_o):
        raise ValueError(f"k_min={k_min} exceeds layer dimensions (n_i={n_i}, n_o={n_o})")
    ratio = math.sqrt(n_o / max(1, n_i))
    k_i = max(k_min, min(n_i, max(1, int(round(math.sqrt(k_total) * ratio)))))
    k_o = max(k_min, min(n_o, max(1, k_total // k_i)))
    best, best_err = (k_i, k_o), abs(k_i * k_o - k_total)
    for di in range(-2, 3):
        for dj in range(-2, 3):
            ci, co = k_i + di, k_o + dj
            if k_min <= ci <= n_i and k_min <= co <= n_o:
                err = abs(ci * co - k_total)
                if err < best_err:
                    best, best_err = (ci, co), err
    if best[0] < k_min or best[1] < k_min:
        raise ValueError(f"Cannot satisfy k_min={k_min} constraints with k_total={k_total}")
    return best


def _generator(device, seed: Optional[int]):
    if seed is None:
        return None
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def init_projection_matrix_gaussian(rows: int, cols: int, dtype: torch.dtype = torch.float32,
                                    device: torch.device = torch.device("cpu"),
                                    seed: Optional[int] = None) -> torch.Tensor:
    """Gaussian JL matrix ``[rows, cols]`` with entries N(0, 1/rows)."""
    P = torch.randn(rows, cols, dtype=dtype, device=device, generator=_generator(device, seed))
    P = P * (1.0 / math.sqrt(rows))
    P.requires_grad_(False)
    return P


def init_projection_matrix_rademacher(rows: int, cols: int, dtype: torch.dtype = torch.float32,
                                      device: torch.device = torch.device("cpu"),
                                      seed: Optional[int] = None) -> torch.Tensor:
    """Entries +-1/sqrt(rows) with equal probability."""
    bits = torch.randint(0, 2, (rows, cols), dtype=torch.int8, device=device,
                         generator=_generator(device, seed))
    P = (bits * 2 - 1).to(dtype) * (1.0 / math.sqrt(rows))
    P.requires_grad_(False)
    return P


def init_projection_matrix_orthonormal(rows: int, cols: int, dtype: torch.dtype = torch.float32,
                                       device: torch.device = torch.device("cpu"),
                                       seed: Optional[int] = None) -> torch.Tensor:
    """Row-orthonormal ``[rows, cols]`` matrix: reduced QR of a float64 Gaussian ``[cols, rows]``."""
    if rows > cols:
        raise ValueError(f"Cannot create {rows} orthonormal rows in {cols} dimensions")
    M = torch.randn(cols, rows, dtype=torch.float64, device=device, generator=_generator(device, seed))
    Q, _ = torch.linalg.qr(M, mode="reduced")
    P = Q.t().to(dtype)
    P.requires_grad_(False)
    return P


def get_projection_initializer(method: str = "gaussian"):
    table = {
        "gaussian": init_projection_matrix_gaussian,
        "rademacher": init_projection_matrix_rademacher,
        "orthonormal": init_projection_matrix_orthonormal,
    }
    if method not in table:
        raise ValueError(f"Unknown projection method: {method}. Choose from {list(table.keys())}")
    return table[method]


def compute_projection_metadata(layer_name: str, layer: nn.Module, k_i: int, k_o: int) -> dict:
    """Per-layer entry of ``metadata.json``."""
    meta = {"name": layer_name, "type": layer.__class__.__name__, "k_i": k_i, "k_o": k_o,
            "k_total": k_i * k_o}
    if hasattr(layer, "weight"):
        shape = layer.weight.shape
        if isinstance(layer, nn.Linear):
            meta["n_o"], meta["n_i"] = shape
        elif isinstance(layer, nn.Conv1d):
            meta["n_o"] = shape[0]
            meta["n_i"] = shape[1] * shape[2]
        elif layer.__class__.__name__ == "Conv1D":
            meta["n_o"], meta["n_i"] = shape
    elif isinstance(layer, nn.Embedding):
        meta["vocab_size"] = layer.num_embeddings
        meta["n_i"] = layer.num_embeddings
        meta["n_o"] = layer.embedding_dim
    return meta


def _find_followed_by_torch():
    """A function that says whether torch follows the operations of this thread one by one (a trace, a dispatch mode, a
    function transform, forward-mode derivatives).  torch answers that only under names of its own; None where it has one of them no more."""
    try:
        tracing, transform = torch._C._get_tracing_state, torch._C._functorch.peek_interpreter_stack
        forward, modes = torch.autograd.forward_ad, torch._C._len_torch_dispatch_stack
        forward._current_level
    except AttributeError:
        return None
    return lambda: modes() > 0 or tracing() is not None or transform() is not None or forward._current_level >= 0


_followed_by_torch = _find_followed_by_torch()


def _bf16_sets_for_kernel(a: torch.Tensor, b: torch.Tensor) -> bool:
    """Whether sets of more than ``ops.SIMILARITY_KERNEL_MAX_ROWS`` rows go through the streaming kernel too.

    Products of bfloat16 values are exact in its float32 sums, so it needs no float32 copies of the rows, and
    no float32 GEMM either (3 x 200 rows of 98304: 7.3 us against 213; 128 x 512 of 4096 8.7 and 87; 512 x 512 of
    98304 339 and 1627; 4096 x 4096 of 4096 715 and 2499; 1 x 512 of 65536 10.6 and 139).  It is taken where its error against 64 bits is no
    larger than the GEMM's: from 96 elements on 0.3 to 1.04 times that, shorter rows 1.0 to 1.3 times (2 x 200 of 64 5.1e-8 and
    4.7e-8); many scores of short rows are the GEMM's by time too (20000 x 20000 of 8: 564 us, in the kernel 793).
    Rows that do not start on 16-byte boundaries are read by element: 512 x 512 of 25871 311 us and 512,
    1024 x 1024 of them 1259 and 1174, so there it ends at 512 rows.  float32 rows stay with the GEMM, which
    takes them as they are; so does what the kernel does not know: gradients, transforms, autocast, sparse
    layouts, lazy negation, shared or overlapping rows."""
    if a.dtype is not torch.bfloat16 or b.dtype is not torch.bfloat16 or a.device != b.device:
        return False
    if any(type(t) is not torch.Tensor or t.layout is not torch.strided or t.is_neg() for t in (a, b)) or a.requires_grad or b.requires_grad \
            or torch.is_autocast_enabled() or torch.are_deterministic_algorithms_enabled() \
            or torch.compiler.is_compiling() or _followed_by_torch is None or _followed_by_torch():
        return False
    dim, rows = a.shape[1], max(a.shape[0], b.shape[0])
    if min(a.shape[0], b.shape[0]) == 0 or dim < 96 or rows > 1 << 16 or a.stride(1) != 1 or b.stride(1) != 1 \
            or min(a.stride(0), b.stride(0)) < dim:
        return False
    aligned = dim % 8 == 0 and all(t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in (a, b))
    return aligned or rows <= 512


def projection_similarity(proj_a: torch.Tensor, proj_b: torch.Tensor) -> torch.Tensor:
    """Gradient-similarity scores ``proj_a @ proj_b.T`` between two sets of projected per-sample
    gradients (``[Na, D]``, ``[Nb, D]`` -> ``[Na, Nb]`` float32): the downstream step of the
    reference's examples (Examples/ghost_gradproj_lm.py:190-196;
    Examples/GradProj_LM/plot_error_with_dim.py:69-86), done while the projections are still on the
    device.  Batch-sized blocks (up to ``ops.SIMILARITY_KERNEL_MAX_ROWS`` rows each: the
    ``[B, total_proj_dim]`` buffers ``collect_batch`` returns) and larger sets of bfloat16 rows
    (:func:`_bf16_sets_for_kernel`) go through the library's streaming kernel; other larger sets are a
    plain dense GEMM and use cuBLAS through torch, in full fp32 so that scores do not depend on the
    TF32 setting.  The kernel's scores may differ in their last bits from call to call, as the parts of a long row are
    added in any order; with ``torch.use_deterministic_algorithms`` the larger sets are the GEMM's.  Host tensors are
    multiplied on the host."""
    if proj_a.shape[-1] != proj_b.shape[-1]:
        raise ValueError("projection sets have different dimensions")
    if proj_a.is_cuda and proj_b.is_cuda and proj_a.dim() == 2 and proj_b.dim() == 2 and \
            (max(proj_a.shape[0], proj_b.shape[0]) <= ops.SIMILARITY_KERNEL_MAX_ROWS or _bf16_sets_for_kernel(proj_a, proj_b)):
        return ops.projection_similarity(proj_a, proj_b)
    a, b = proj_a.float(), proj_b.float()
    if a.is_cuda:
        prev = torch.backends.cuda.matmul.allow_tf32
        torch.backends.cuda.matmul.allow_tf32 = False
        try:
            return a @ b.t()
        finally:
            torch.backends.cuda.matmul.allow_tf32 = prev
    return a @ b.t()

"""Parity of every CUDA kernel (called through the C ABI) against the CPU oracle."""
import numpy as np
import pytest
import torch

from conftest import as_dtype
from oracle import ghost_oracle as O

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-4, torch.bfloat16: 2e-2}   # relative Frobenius, per the north star


def ops():
    from ghostsuite_b200 import ops as _ops
    return _ops


def make(N, T, d, p, dtype, seed=0):
    g = torch.Generator().manual_seed(seed)
    A = (torch.randn(N, T, d, generator=g) / d ** 0.5).to(dtype)
    G = (torch.randn(N, T, p, generator=g) / p ** 0.5).to(dtype)
    return A, G


def after():
    from ghostsuite_b200 import _lib
    torch.cuda.synchronize()
    _lib.poll_kernel_error()


LIN_CASES = [
    # n_train, n_val, T, d, p
    (5, 3, 6, 16, 24),        # several samples per tile, ragged everything
    (64, 16, 1, 512, 1024),   # MLP config: T = 1
    (3, 1, 130, 72, 40),      # T just above one tile, single validation sample
    (2, 2, 300, 200, 136),    # validation rows straddle the 256-wide tile
    (4, 2, 128, 64, 64),      # exactly tile-aligned
    (2, 3, 37, 10, 50),       # feature sizes that are not multiples of 8
    (33, 20, 9, 64, 264),     # 17..32 validation samples share one streaming pass; two train blocks
    (40, 35, 20, 72, 136),    # more than 32 validation samples: two passes over the train tiles
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", LIN_CASES)
def test_gram_dot(case, dtype):
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype)
    M = ops().gram_dot(A.cuda(), G.cuda(), n_v)
    after()
    ref = O.linear_dot_exact(A, G, n_v)
    assert M.shape == (n_v, n_t)
    assert O.rel_fro(M, ref) < TOL[dtype]


# token counts on both sides of what chooses the tile shape: one tile of 128 x 128, fewer tiles of 256 x 256 than CTA
# pairs, a full round of them; both operands and their sums through the layer's hook, which shares their copies
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(2, 1, 17, 63, 65), (5, 4, 64, 130, 64), (4, 2, 512, 96, 72), (40, 10, 100, 64, 200), (300, 40, 31, 65, 70)])
@pytest.mark.parametrize("in_by_out", [False, True])
def test_gram_hook_tile_shapes(in_by_out, case, dtype):
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=33)
    M, grad, sums, _, _ = ops().dense_hook(A.cuda(), G.cuda(), n_v, in_by_out, True, torch.float32, 0.5, True, torch.float32, False, True)
    after()
    S = torch.einsum("ntp,ntd->npd", G.cuda().double(), A.cuda().double()).flatten(1)
    ref, gref = S[n_t:] @ S[:n_t].t(), 0.5 * S[:n_t].sum(0).view(p, d)
    # entries cancel over the token pairs: errors are relative to the norms of the pair's gradients.  float32 carries two
    # parts of 8 bits; a Gram entry sums d (p) products in float32 that the tensor core truncates
    tol = (2 * 2.0 ** -16 if dtype == torch.float32 else 0.) + max(d, p) * 2.0 ** -23
    scale = (A.cuda().double().flatten(1).norm(dim=1) * G.cuda().double().flatten(1).norm(dim=1))
    assert ((M.double() - ref).abs() <= tol * scale[n_t:, None] * scale[None, :n_t]).all()
    assert O.rel_fro(grad if not in_by_out else grad.t(), gref) < 2 * 2.0 ** -16 + T * n_t * 2.0 ** -23
    assert O.rel_fro(sums, G.double().sum(1)) < 1e-6


# calls of few tiles and long rows, whose tiles are shared by clusters: K steps of both operands that part inside a CTA's run, at its
# edge and leave most CTAs one operand only; columns and rows that end inside a quarter, one token, more tiles than clusters of eight; a
# sample a lane, several a warp, two and one, and warps without rows
@pytest.mark.parametrize("dtype,mode", [(torch.bfloat16, 0), (torch.float32, 0), (torch.bfloat16, 1)])
@pytest.mark.parametrize("case", [(2, 1, 1, 2048, 2048), (5, 3, 13, 4096, 40), (3, 2, 70, 24, 5003), (9, 5, 41, 1031, 1500), (33, 4, 64, 1536, 1536),
                                  (70, 9, 1, 3000, 64), (43, 3, 3, 64, 2500), (8, 2, 32, 1600, 300), (7, 3, 31, 900, 1800), (5, 2, 129, 2048, 64)])
def test_gram_tiles_shared_by_clusters(case, dtype, mode):
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=34)
    from ghostsuite_b200 import _lib
    assert _lib.load().ghost_gram_cluster_size(2 if dtype == torch.float32 else 1, n_t, n_v, T, d, p) > 1
    M = ops().gram_dot(A.cuda(), G.cuda(), n_v, round_mode=mode)
    after()
    a, g = A.cuda().double(), G.cuda().double()
    S = torch.einsum("ntp,ntd->npd", g, a).flatten(1)
    # as in test_gram_hook_tile_shapes; a rounded Gram entry and product are within 2^-8 of themselves each, no longer relative to a pair
    # that cancels but to the token pairs' products
    tol = (2 * 2.0 ** -16 if dtype == torch.float32 else 0.) + max(d, p) * 2.0 ** -23
    scale = a.flatten(1).norm(dim=1) * g.flatten(1).norm(dim=1)
    bound = tol * scale[n_t:, None] * scale[None, :n_t]
    if mode:
        ga = torch.einsum("vsd,btd->vbst", a[n_t:], a[:n_t]) * torch.einsum("vsp,btp->vbst", g[n_t:], g[:n_t])
        bound = bound + 3 * 2.0 ** -8 * ga.abs().sum((2, 3))
    assert ((M.double() - S[n_t:] @ S[:n_t].t()).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(5, 3, 130, 72, 40), (4, 2, 256, 128, 64), (9, 2, 300, 200, 136),
                                  (700, 300, 1, 64, 48), (3, 5, 513, 96, 256)])
def test_gram_dot_cta_pair_kernel(case, dtype):
    """The cta_group::2 variant (256 x 256 tile per CTA pair) against the oracle and the
    single-CTA kernel, including ragged tiles and an odd number of tiles."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=21)
    ref = O.linear_dot_exact(A, G, n_v) if n_t * n_v < 5000 else None
    try:
        _lib.check(lib.ghost_set_gram_pair_mode(2))
        M2 = ops().gram_dot(A.cuda(), G.cuda(), n_v)
        after()
        _lib.check(lib.ghost_set_gram_pair_mode(0))
        M1 = ops().gram_dot(A.cuda(), G.cuda(), n_v)
        after()
    finally:
        _lib.check(lib.ghost_set_gram_pair_mode(1))
    assert O.rel_fro(M2, M1.cpu()) < 1e-5
    if ref is not None:
        assert O.rel_fro(M2, ref) < TOL[dtype]


def test_gram_dot_reference_rounding_mode():
    """round_mode=1 reproduces the reference's bf16-rounded Grams (vector = column sums)."""
    n_t, n_v, T, d, p = 5, 3, 6, 16, 24
    A, G = make(n_t + n_v, T, d, p, torch.bfloat16, seed=3)
    M = ops().gram_dot(A.cuda(), G.cuda(), n_v, round_mode=1)
    after()
    ref = O.linear_dot_reference(A, G, n_v, use_ghost=True)
    assert O.rel_fro(M.sum(0), ref) < 2e-3


def test_gram_dot_golden(golden):
    for tag, dt in (("f32", torch.float32), ("bf16", torch.bfloat16)):
        A = as_dtype(golden[f"lin_{tag}_A"], tag)
        G = as_dtype(golden[f"lin_{tag}_G"], tag)
        M = ops().gram_dot(A.cuda(), G.cuda(), 3)
        after()
        rows = torch.from_numpy(golden[f"lin_{tag}_rows_materialised"])
        assert O.rel_fro(M, rows) < TOL[dt]
        assert O.rel_fro(M.sum(0), torch.from_numpy(golden[f"lin_{tag}_nv3_ghost1_w"])) < 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", LIN_CASES)
def test_wgrad(case, dtype):
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=1)
    N = n_t + n_v
    scale = N / n_t
    out = ops().wgrad(G[:n_t].cuda(), A[:n_t].cuda(), scale, dtype)        # Linear layout [p, d]
    outc = ops().wgrad(A[:n_t].cuda(), G[:n_t].cuda(), scale, dtype)       # Conv1D layout [d, p]
    after()
    ref = torch.einsum("btp,btd->pd", G[:n_t].double(), A[:n_t].double()) * scale
    assert out.shape == (p, d) and out.dtype == dtype
    tol = 1e-4 if dtype == torch.float32 else 1e-2
    assert O.rel_fro(out, ref) < tol
    assert O.rel_fro(outc, ref.t()) < tol
    # against the reference formula in its own dtype
    ref2 = O.linear_train_grad(A, G * N, n_v)
    assert O.rel_fro(out, ref2) < (1e-4 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("case", [(70, 64, 128), (130 * 3, 192, 320), (2700, 448, 64), (5000, 768, 1024),
                                  (64 * 300, 128, 384), (9, 64, 64)])
def test_wgrad_cta_pair_kernel(case):
    """The CTA-pair split-K pass (mode 2: wherever the column counts are multiples of 64, odd tile
    counts included) against the single-CTA pass and the fp64 contraction."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    rows, d, p = case
    A, G = make(1, rows, d, p, torch.bfloat16, seed=23)
    ref = torch.einsum("btp,btd->pd", G.double(), A.double())
    res = {}
    try:
        for mode in (0, 2):
            _lib.check(lib.ghost_set_wgrad_pair_mode(mode))
            res[mode] = ops().wgrad(G.cuda(), A.cuda(), 1.0, torch.float32)
            after()
    finally:
        _lib.check(lib.ghost_set_wgrad_pair_mode(1))
    assert O.rel_fro(res[2], ref) < 1e-2
    assert O.rel_fro(res[2], res[0].cpu()) < 1e-5      # same products, another order of fp32 additions


def test_wgrad_accumulate():
    A, G = make(6, 40, 64, 48, torch.bfloat16, seed=5)
    o = ops()
    base = torch.randn(48, 64).to(torch.float32).cuda()
    out = base.clone()
    o.wgrad(G.cuda(), A.cuda(), 0.5, torch.float32, out=out, accumulate=True)
    after()
    ref = base.cpu().double() + 0.5 * torch.einsum("btp,btd->pd", G.double(), A.double())
    assert O.rel_fro(out, ref) < 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", LIN_CASES)
def test_persample_dot(case, dtype):
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=2)
    N = n_t + n_v
    M, grad = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=N / n_t,
                                  grad_dtype=dtype)
    after()
    ref = O.linear_dot_exact(A, G, n_v)
    assert O.rel_fro(M, ref) < TOL[dtype]
    gref = torch.einsum("btp,btd->pd", G[:n_t].double(), A[:n_t].double()) * (N / n_t)
    assert O.rel_fro(grad, gref) < (1e-4 if dtype == torch.float32 else 1e-2)
    # both paths agree with each other far inside the tolerance
    M2 = ops().gram_dot(A.cuda(), G.cuda(), n_v)
    after()
    assert O.rel_fro(M, M2.cpu()) < TOL[dtype]


@pytest.mark.parametrize("case", [(5, 3, 6, 16, 24), (3, 1, 130, 72, 40), (2, 2, 300, 200, 136), (9, 4, 70, 264, 520),
                                  # column counts that take the CTA-pair kernel (multiples of 64, an even
                                  # number of 128-row tiles), T not a multiple of 32
                                  (5, 3, 130, 256, 512), (3, 2, 77, 768, 256), (4, 2, 1024, 512, 1024)])
@pytest.mark.parametrize("which", ["X", "Y"])
def test_persample_dot_column_sums(case, which):
    """Per-sample column sums of one operand taken inside the GEMM pass (the bias terms)."""
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, torch.bfloat16, seed=13)
    M, grad, cs = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=1.0,
                                      grad_dtype=torch.float32, colsum_of=which)
    after()
    src = G if which == "X" else A
    assert cs.shape == (n_t + n_v, src.shape[-1])
    assert O.rel_fro(cs, src.double().sum(1)) < 1e-5
    assert O.rel_fro(M, O.linear_dot_exact(A, G, n_v)) < 2e-2
    # fp32 operands reach the kernel as a bf16 hi/lo split: no fused sums
    res = ops().persample_dot(G.float().cuda(), A.float().cuda(), n_v, colsum_of=which)
    assert res[2] is None


# token counts around a step of 16, a stage of 32 / 64 and one of 128; columns around a panel of 64, one and two
# tiles of 128; every operand needs a copy, so the padded and the two-part layouts are what runs
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(3, 2, 1, 63, 65), (2, 1, 16, 127, 129), (3, 1, 17, 257, 63), (2, 2, 33, 130, 70),
                                  (2, 1, 63, 65, 257), (2, 1, 129, 300, 140), (33, 3, 5, 71, 199), (2, 1, 260, 190, 510),
                                  # chunks of 64 rows that add up their sums as a cluster of two to eight, and more of them
                                  (1, 1, 65, 70, 130), (2, 1, 300, 129, 66), (1, 2, 512, 64, 300), (1, 1, 513, 33, 72)])
def test_padded_and_split_operands(case, dtype):
    """Padded bf16 copies and two-part float32 operands: matrix, train gradient, column sums, and the
    gradient GEMM with results that no 16-byte store fits, through both tile kernels."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=31)
    # values and residuals are 8 bits each and the product of two residuals is left out: 2^-16 a product, and
    # the bf16 path stores its tiles in 8 bits
    tol = 2 * 2.0 ** -16 if dtype == torch.float32 else 2 * 2.0 ** -8
    S = torch.einsum("ntp,ntd->npd", G.double(), A.double())
    ref, gref, cref = torch.einsum("vpd,bpd->vb", S[n_t:], S[:n_t]), S[:n_t].sum(0), G.double().sum(1)
    size = (S[n_t:].flatten(1).norm(dim=1)[:, None] * S[:n_t].flatten(1).norm(dim=1)[None]).norm()
    old = torch.full((p, d), 0.25, dtype=dtype, device="cuda")
    try:
        for mode in (0, 2):
            _lib.check(lib.ghost_set_persample_pair_mode(mode))
            _lib.check(lib.ghost_set_wgrad_pair_mode(mode))
            M, grad, sums = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=0.5,
                                                grad_dtype=torch.float32, colsum_of="X")
            hook = ops().dense_hook(A.cuda(), G.cuda(), n_v, False, False, torch.float32, 0.5, True, torch.float32,
                                    False, True)
            out = ops().wgrad(G[:n_t].cuda(), A[:n_t].cuda(), 0.5, dtype)
            acc = ops().wgrad(G[:n_t].cuda(), A[:n_t].cuda(), 0.5, dtype, out=old.clone(), accumulate=True)
            after()
            assert (M.cpu().double() - ref).norm() < tol * size
            assert O.rel_fro(grad, 0.5 * gref) < tol
            assert (hook[0].cpu().double() - ref).norm() < tol * size and O.rel_fro(hook[1], 0.5 * gref) < tol
            for got in ([sums] if sums is not None else []) + [hook[2]]:
                assert O.rel_fro(got, cref) < 1e-6
            assert O.rel_fro(out, 0.5 * gref) < tol
            assert O.rel_fro(acc.float() - 0.25, 0.5 * gref) < tol + 2 * 0.25 * (p * d) ** 0.5 / gref.norm() * (
                2.0 ** -24 if dtype == torch.float32 else 2.0 ** -9) * 2
    finally:
        _lib.check(lib.ghost_set_persample_pair_mode(1))
        _lib.check(lib.ghost_set_wgrad_pair_mode(1))


# sample counts around the streaming pass's blocks: 4, 8, 16, 32 validation and 8, 16, 32 train rows a stage; a budget of
# 1 MiB makes groups of single samples, whose sums go through the workspace
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(1, 1, 3, 5, 7), (8, 4, 3, 70, 130), (9, 5, 2, 300, 129), (16, 8, 3, 257, 33), (17, 9, 2, 513, 20),
                                  (32, 16, 2, 256, 128), (33, 17, 2, 130, 140), (70, 33, 1, 40, 300), (40, 3, 4, 700, 260)])
def test_streaming_pass_blocks(case, dtype):
    """Whole numbers whose products and sums float32 holds, and whose tiles bf16 does: equal in any order of addition."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    n_t, n_v, T, d, p = case
    g = torch.Generator().manual_seed(n_t)
    A, G = (torch.randint(-2, 3, (n_t + n_v, T, c), generator=g).to(dtype) for c in (d, p))
    S = torch.einsum("ntp,ntd->npd", G.double(), A.double())
    ref, gref = torch.einsum("vpd,bpd->vb", S[n_t:], S[:n_t]), S[:n_t].sum(0)
    assert S.abs().max() <= 256 and S[n_t:].flatten(1).norm(dim=1).max() * S[:n_t].flatten(1).norm(dim=1).max() < 2 ** 24
    try:
        for budget in (12 << 30, 1 << 20):
            _lib.check(lib.ghost_set_persample_budget_bytes(budget))
            M, grad = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=0.5, grad_dtype=torch.float32)[:2]
            after()
            assert torch.equal(M.cpu().double(), ref) and torch.equal(grad.cpu().double(), 0.5 * gref)
            half = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=0.5, grad_dtype=torch.bfloat16)[1]
            after()
            assert torch.equal(half.cpu(), (0.5 * gref).bfloat16())          # summed in float32, rounded once
    finally:
        _lib.check(lib.ghost_set_persample_budget_bytes(12 << 30))


@pytest.mark.parametrize("sizes", [(37, 11, 70, 136, 264), (70, 35, 12, 72, 264)])
def test_persample_dot_in_groups(sizes):
    """A small workspace budget forces the train samples through in several groups (and several
    validation / train blocks of the streaming kernel): same numbers as the single-pass run."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    n_t, n_v, T, d, p = sizes
    A, G = make(n_t + n_v, T, d, p, torch.bfloat16, seed=11)
    ref = O.linear_dot_exact(A, G, n_v)
    gref = torch.einsum("btp,btd->pd", G[:n_t].double(), A[:n_t].double())
    try:
        for budget in (12 << 30, 2 << 20):
            _lib.check(lib.ghost_set_persample_budget_bytes(budget))
            M, grad, cs = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=1.0,
                                              grad_dtype=torch.float32, colsum_of="X")
            after()
            assert O.rel_fro(M, ref) < 2e-2
            assert O.rel_fro(grad, gref) < 1e-2
            assert O.rel_fro(cs, G.double().sum(1)) < 1e-5
    finally:
        _lib.check(lib.ghost_set_persample_budget_bytes(12 << 30))


@pytest.mark.parametrize("case", [(5, 3, 70, 64, 128), (3, 1, 130, 192, 320), (9, 4, 300, 448, 64),
                                  (4, 2, 64, 768, 1024), (33, 20, 9, 64, 256), (37, 11, 70, 128, 384)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_persample_dot_cta_pair_kernel(case, dtype):
    """The CTA-pair tile pass (mode 2: wherever the column counts allow it, odd tile counts and
    several train groups included) stores the same tiles as the single-CTA pass: identical train
    gradient, and dot products equal up to the order of the fp32 additions."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, dtype, seed=17)
    res = {}
    try:
        _lib.check(lib.ghost_set_persample_budget_bytes(8 << 20))
        for mode in (0, 2):
            _lib.check(lib.ghost_set_persample_pair_mode(mode))
            res[mode] = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=1.0,
                                            grad_dtype=torch.float32)[:2]
            after()
    finally:
        _lib.check(lib.ghost_set_persample_pair_mode(1))
        _lib.check(lib.ghost_set_persample_budget_bytes(12 << 30))
    assert torch.equal(res[0][1], res[2][1])
    assert O.rel_fro(res[2][0], res[0][0].cpu()) < 1e-5
    assert O.rel_fro(res[2][0], O.linear_dot_exact(A, G, n_v)) < TOL[dtype]
    assert lib.ghost_set_persample_pair_mode(3) < 0


# edges of the float32 streaming kernel: 8- and 16-row validation blocks, 32-row train blocks, weights that
# end inside a tile, train groups that add up over several launches
@pytest.mark.parametrize("case", [(1, 1, 3, 1), (32, 8, 129, 255), (33, 9, 127, 257), (5, 17, 1, 300), (70, 16, 130, 40)])
@pytest.mark.parametrize("grad_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("budget", [12 << 30, 3 << 20])
def test_persample_float32_tiles_exact(case, grad_dtype, budget):
    """Small whole numbers: every product and partial sum is a whole number below 2^24, so the float32
    results are exact whatever the order of the additions; the bf16 gradient is one rounding of it."""
    from ghostsuite_b200 import _lib
    n_t, n_v, p, d = case
    gen = torch.Generator().manual_seed(sum(case))
    A = torch.randint(-3, 4, (n_t + n_v, 5, d), generator=gen).float()
    G = torch.randint(-3, 4, (n_t + n_v, 5, p), generator=gen).float()
    per = torch.einsum("ntp,ntd->npd", G.double(), A.double())
    want = per[n_t:].flatten(1) @ per[:n_t].flatten(1).T
    lib = _lib.load()
    try:
        _lib.check(lib.ghost_set_persample_budget_bytes(budget))
        M, grad = ops().persample_dot(G.cuda(), A.cuda(), n_v, want_grad=True, grad_scale=1.0, grad_dtype=grad_dtype)
        after()
    finally:
        _lib.check(lib.ghost_set_persample_budget_bytes(12 << 30))
    assert torch.equal(M.cpu().double(), want)
    assert torch.equal(grad.cpu(), per[:n_t].sum(0).to(grad_dtype))


@pytest.mark.parametrize("case", [(5, 8, 70, 64, 128), (12, 8, 64, 256, 512), (7, 16, 33, 192, 320),
                                  (33, 4, 40, 72, 264), (3, 32, 20, 128, 256)])
def test_tile_pass_and_gathered_tile_dot(case):
    """The per-sample path as two calls with the validation tiles laid out as an all-gather over
    ranks leaves them ([ranks][tiles][per rank][128 x 256]): every split of the validation batch
    gives the matrix and the train gradient of the one-call path (same tiles, same kernel)."""
    n_t, n_v, T, d, p = case
    A, G = make(n_t + n_v, T, d, p, torch.bfloat16, seed=50 + n_v)
    Ac, Gc = A.cuda(), G.cuda()
    o = ops()
    gdt = torch.float32 if n_t > 32 else torch.bfloat16
    M_ref, grad_ref, cs_ref = o.persample_dot(Gc, Ac, n_v, dot_scale=1.5, want_grad=True, grad_scale=0.25,
                                              grad_dtype=gdt, colsum_of="X")
    after()
    block = 8 if n_v <= 8 else (16 if n_v <= 16 else 32)
    for ranks in (1, 2, 4, 8):
        per = n_v // ranks
        if per * ranks != n_v or per == 0:
            continue
        assert block % per == 0 or per % block == 0
        cs = torch.full((n_t + n_v, p), float("nan"), device="cuda")
        V = torch.stack([o.persample_tiles(Gc, Ac, n_t + r * per, per, "X", cs) for r in range(ranks)])
        W = o.persample_tiles(Gc, Ac, 0, n_t, "X", cs)
        M, grad = o.tile_dot(V, W, p, d, dot_scale=1.5, want_grad=True, grad_scale=0.25, grad_dtype=gdt)
        after()
        assert O.rel_fro(M, M_ref.cpu()) < 1e-5, ranks
        assert torch.equal(grad, grad_ref), ranks
        assert O.rel_fro(cs, cs_ref.double().cpu()) < 1e-6, ranks
    # a split that does not fit the kernel's blocks of validation rows is refused, not mangled
    if n_v == 16:
        V = torch.zeros(4, W.shape[0], 3, 32768, dtype=torch.bfloat16, device="cuda")      # 12 = 4 x 3
        with pytest.raises(ValueError):
            o.tile_dot(V, W, p, d)
        class FourRanks:
            world = 4

            @staticmethod
            def gather_rows(t):
                return t.repeat(4, 1, 1, 1)

        assert o.persample_dot_exchanged(Gc[:n_t + 3], Ac[:n_t + 3], 3, FourRanks) is None
        res = o.persample_dot_exchanged(Gc[:n_t + 4], Ac[:n_t + 4], 4, FourRanks, want_grad=True,
                                        grad_dtype=torch.float32, colsum_of="X")
        after()
        one = o.persample_dot(Gc[:n_t + 4], Ac[:n_t + 4], 4, want_grad=True, grad_dtype=torch.float32, colsum_of="X")
        # four "ranks" that all hold the same four validation samples: the local block four times
        assert res[0].shape == (16, n_t) and O.rel_fro(res[0], one[0].repeat(4, 1).cpu()) < 1e-5
        assert torch.equal(res[1], one[1]) and O.rel_fro(res[2], one[2].double().cpu()) < 1e-6


# both sides of the split-K rule: one CTA per tile stores the result, many add into the workspace
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,m,n", [(20000, 64, 128), (20000, 72, 40), (300, 256, 520), (130, 37, 264)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_wgrad_direct_and_split(rows, m, n, dtype, out_dtype):
    g = torch.Generator().manual_seed(17)
    X, Y = (torch.randn(1, rows, c, generator=g).to(dtype).cuda() for c in (m, n))
    out = ops().wgrad(X, Y, 0.25, out_dtype)
    ref = 0.25 * X[0].double().t() @ Y[0].double()
    after()
    tol = 1e-4 if dtype == torch.float32 else 1e-5          # hi/lo parts; exact products
    assert O.rel_fro(out, ref) < (3e-3 if out_dtype == torch.bfloat16 else tol)       # 2^-9 of rounding
    more = ops().wgrad(X, Y, 0.25, out_dtype, out=out.clone(), accumulate=True)
    after()
    assert O.rel_fro(more, out.double() + ref) < (6e-3 if out_dtype == torch.bfloat16 else tol)


# tokens and features on both sides of the 64 x 64 tile, windows that overhang the input, every option
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("use_gram", [False, True])
@pytest.mark.parametrize("case", [(3, 2, 4, 9, 7, 5, (3, 3), (1, 1), (1, 1), (1, 1)),
                                  (4, 1, 3, 12, 11, 8, (5, 3), (2, 1), (2, 0), (1, 1)),
                                  (2, 2, 7, 10, 13, 70, (3, 2), (1, 2), (2, 1), (2, 3)),
                                  (5, 3, 65, 8, 8, 24, (1, 1), (1, 1), (0, 0), (1, 1))])
def test_conv_hook(case, use_gram, dtype):
    n_t, n_v, C, H, W, p, k, stride, pad, dil = case
    N = n_t + n_v
    g = torch.Generator().manual_seed(19)
    A = torch.randn(N, C, H, W, generator=g).to(dtype)
    tok = torch.nn.functional.unfold(A.double(), k, dilation=dil, padding=pad, stride=stride).transpose(1, 2)
    Ho = (H + 2 * pad[0] - dil[0] * (k[0] - 1) - 1) // stride[0] + 1
    B = torch.randn(N, p, Ho, tok.shape[1] // Ho, generator=g).to(dtype)
    Bt = B.double().reshape(N, p, -1).transpose(1, 2)
    M, grad, sums, _, _ = ops().conv_hook(A.cuda(), B.cuda(), n_v, (*k, *stride, *pad, *dil), use_gram, torch.float32, 0.5,
                                          True, torch.float32)
    after()
    per = torch.einsum("ntp,ntd->npd", Bt, tok).reshape(N, -1)
    assert O.rel_fro(M, per[n_t:] @ per[:n_t].t()) < TOL[dtype]
    assert O.rel_fro(grad.reshape(-1), 0.5 * per[:n_t].sum(0)) < (1e-4 if dtype == torch.float32 else 1e-2)
    assert O.rel_fro(sums, Bt.sum(1)) < 1e-5


# a window whose padding alone needs 64-bit offsets; bias sums behind one block of positions and behind many
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("use_gram", [False, True])
@pytest.mark.parametrize("case", [(2, 1, 3, 2, 2, 5, (1, 1), (20000, 20000), (20000, 20000), (1, 1)),
                                  (2, 1, 2, 40, 40, 130, (3, 3), (1, 1), (1, 1), (1, 1))])
def test_conv_operands_in_one_launch(case, use_gram, dtype):
    test_conv_hook(case, use_gram, dtype)


def test_conv_operands_beyond_one_grid():
    """More blocks of features than a grid has rows: an operand a launch, the bytes of the single-operand entry."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    C, p, N = 65535 * 64, 70, 2
    A, B = torch.randn(N, C, 1, 1).cuda(), torch.randn(N, p, 1, 1).cuda()
    st = torch.cuda.current_stream().cuda_stream
    got = [torch.zeros(N, 2, 1, w, dtype=torch.bfloat16, device="cuda") for w in (C, 128)]
    sums = torch.zeros(N, p, device="cuda")
    _lib.check(lib.ghost_conv_operands(A.data_ptr(), 1, B.data_ptr(), 1, N, C, 1, 1, 1, 1, 1, 1, 0, 0, 1, 1, p, 1, 1, 2, 0,
                                       got[0].data_ptr(), got[1].data_ptr(), sums.data_ptr(), st))
    for x, c, out in ((A, C, got[0]), (B, p, got[1])):
        want = torch.zeros_like(out)
        _lib.check(lib.ghost_conv_tokens_bf16(x.data_ptr(), 1, N, c, 1, 1, 1, 1, 1, 1, 0, 0, 1, 1, want.data_ptr(), out.shape[3],
                                              out.shape[3], 2, 0, 1, 0, 1, st))
        after()
        assert torch.equal(out, want)
        # hi + lo: 2^-9 of the value is left to lo, which is rounded to 2^-9 of itself
        assert ((out.float().sum(1)[:, 0, :c] - x[:, :, 0, 0]).abs() <= 2.0 ** -17 * x[:, :, 0, 0].abs()).all()
    assert torch.equal(sums, B[:, :, 0, 0])


# edges of the one-launch kernel: T on both sides of its 8 x 4 token tile and of whole-sample groups,
# one sample, widths off and on its 64 / 128 / 1024 column units, odd widths (no 16-byte loads)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(1, 1, 1, 1, 1), (64, 16, 1, 512, 1024), (9, 9, 1, 130, 67), (5, 3, 2, 64, 1028),
                                  (3, 5, 3, 33, 65), (4, 3, 4, 128, 64), (2, 2, 7, 40, 200), (3, 2, 8, 260, 12),
                                  (2, 3, 9, 68, 1025), (5, 2, 16, 100, 36)])
@pytest.mark.parametrize("in_by_out", [False, True])
def test_dense_small(case, dtype, in_by_out):
    o = ops()
    n_t, n_v, T, d, p = case
    g = torch.Generator().manual_seed(31)
    A = (torch.randn(n_t + n_v, T, d, generator=g) / d ** 0.5).to(dtype)
    B = (torch.randn(n_t + n_v, T, p, generator=g) / p ** 0.5).to(dtype)
    from ghostsuite_b200 import _lib
    assert _lib.load().ghost_dense_small_fits(int(dtype == torch.float32), n_t, n_v, T, d, p) == 1
    l0 = _lib.launch_count()
    M, grad, sums, Mb, sb = o.dense_hook(A.cuda(), B.cuda(), n_v, in_by_out, True, torch.float32, 0.5, True, torch.float32)
    assert _lib.launch_count() - l0 == 1
    after()
    # float32 sums of exact products of the given values
    assert O.rel_fro(M, O.linear_dot_exact(A, B, n_v)) < 1e-5
    ref = 0.5 * torch.einsum("btp,btd->pd", B[:n_t].double(), A[:n_t].double())
    assert O.rel_fro(grad, ref.t() if in_by_out else ref) < 1e-5
    assert O.rel_fro(sums, B.double().sum(1)) < 1e-5
    assert Mb.shape == (n_v, n_t) and sb.shape == (p,)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(8, 6, 24), (12, 1, 10), (5, 300, 520), (3, 1024, 768),
                                   (3, 65, 300), (4, 129, 24), (3, 2000, 40), (40, 449, 513)])
def test_colsum_and_bias(shape, dtype):
    N, T, p = shape
    g = torch.Generator().manual_seed(4)
    G = torch.randn(N, T, p, generator=g).to(dtype)
    o = ops()
    cs = o.colsum(G.cuda())
    n_v = 2
    M = o.small_gram(cs, n_v)
    bgrad = o.rows_sum(cs, N - n_v, N / (N - n_v), dtype)
    after()
    ref = G.double().sum(1)
    assert O.rel_fro(cs, ref) < 1e-5
    assert O.rel_fro(M, O.bias_dot_exact(G, n_v)) < 1e-4
    assert O.rel_fro(bgrad, O.bias_train_grad((G * N).clone(), n_v)) < (1e-5 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(8, 6, 16), (5, 70, 768), (4, 33, 1024), (3, 9, 20), (2, 5, 1536)])
def test_layernorm(shape, dtype):
    N, T, F = shape
    g = torch.Generator().manual_seed(6)
    A = (torch.randn(N, T, F, generator=g) * 1.5 + 0.3).to(dtype)
    G = (torch.randn(N, T, F, generator=g) / F ** 0.5).to(dtype)
    gw, gb = ops().layernorm_persample(A.cuda(), G.cuda(), 1e-5)
    after()
    rw, rb = O.layernorm_persample_exact(A, G, 1e-5)
    assert O.rel_fro(gw, rw) < 1e-4
    assert O.rel_fro(gb, rb) < 1e-4


def test_layernorm_golden(golden):
    eps = float(golden["ln_eps"][0])
    for tag in ("f32", "bf16"):
        A = as_dtype(golden[f"ln_{tag}_A"], tag)
        G = as_dtype(golden[f"ln_{tag}_G"], tag)
        o = ops()
        gw, gb = o.layernorm_persample(A.cuda(), G.cuda(), eps)
        Mw, Mb = o.small_gram(gw, 3), o.small_gram(gb, 3)
        after()
        assert O.rel_fro(Mw.sum(0), torch.from_numpy(golden[f"ln_{tag}_nv3_w"])) < 2e-2
        assert O.rel_fro(Mb.sum(0), torch.from_numpy(golden[f"ln_{tag}_nv3_b"])) < 2e-2
        tw = o.rows_sum(gw, 5, 8 / 5, torch.float32)
        after()
        assert O.rel_fro(tw, torch.from_numpy(golden[f"ln_{tag}_train_grad_w"])) < (1e-5 if tag == "f32" else 2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(5, 3, 6, 8, 11), (4, 2, 64, 40, 50), (3, 2, 100, 768, 7), (6, 1, 33, 16, 1000),
                                  # tables that span several 4096-id tiles of the bucket scan, feature counts
                                  # off the 16-byte path, a crowded row in the last, partial tile
                                  (6, 2, 700, 20, 9001), (40, 2, 64, 72, 4099), (12, 3, 50, 264, 12289)])
def test_embedding(case, dtype):
    n_t, n_v, T, d, vocab = case
    N = n_t + n_v
    g = torch.Generator().manual_seed(8)
    ids = torch.randint(0, vocab, (N, T), generator=g)
    if vocab > 4096:
        ids[:, :3] = vocab - 1
        ids[:, 3] = 4095
        ids[:, 4] = 4096
    G = (torch.randn(N, T, d, generator=g) / d ** 0.5).to(dtype)
    o = ops()
    M = o.embedding_dot(ids.cuda(), G.cuda(), n_v, vocab)
    grad = o.embedding_wgrad(ids.cuda(), G.cuda(), n_t, vocab, float(N), float(n_t))
    after()
    assert O.rel_fro(M, O.embedding_dot_exact(ids, G, n_v)) < (1e-5 if dtype == torch.float32 else 1e-4)
    ref = O.embedding_train_grad(ids, G * N, n_v, vocab, sequential=True)
    # index / gather work: bit-exact against the CPU sequential order
    assert torch.equal(grad.cpu().float(), ref.float())


# the join's items cut into ranges of features: widths on and off the 128 features of a cut and of the 16-byte loads, one
# cut or many, an infinite entry in one of them, hot ids
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [128, 136, 701, 2056, 4224])
@pytest.mark.parametrize("n_t,n_v,T,vocab", [(3, 2, 20, 7), (2, 2, 200, 3)])
def test_embedding_dot_of_few_items(n_t, n_v, T, vocab, d, dtype):
    g = torch.Generator().manual_seed(12)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=g)
    G = (torch.randn(n_t + n_v, T, d, generator=g) / d ** 0.5).to(dtype)
    M = ops().embedding_dot(ids.cuda(), G.cuda(), n_v, vocab)
    after()
    assert O.rel_fro(M, O.embedding_dot_exact(ids, G, n_v)) < (1e-5 if dtype == torch.float32 else 1e-4)
    G[0, 0], G[0, 0, d - 1] = 0, float("inf")              # sample 0's row of one id: an infinity in the last range
    G[n_t:, :, d - 1] = 1
    ids[n_t:, 0] = ids[0, 0]
    M = ops().embedding_dot(ids.cuda(), G.cuda(), n_v, vocab)
    after()
    assert (M[:, 0] == float("inf")).all() and torch.isfinite(M[:, 1:]).all()


def test_embedding_position_ids_and_golden(golden):
    # position-embedding pattern: every sample has ids 0..T-1 (all buckets hold n_train tokens)
    n_t, n_v, T, d = 40, 2, 16, 24
    ids = torch.arange(T).repeat(n_t + n_v, 1)
    G = torch.randn(n_t + n_v, T, d, generator=torch.Generator().manual_seed(1))
    o = ops()
    M = o.embedding_dot(ids.cuda(), G.cuda(), n_v, T)
    grad = o.embedding_wgrad(ids.cuda(), G.cuda(), n_t, T, float(n_t + n_v), float(n_t))
    after()
    assert O.rel_fro(M, O.embedding_dot_exact(ids, G, n_v)) < 1e-5
    assert torch.equal(grad.cpu(), O.embedding_train_grad(ids, G * (n_t + n_v), n_v, T))
    ids = torch.from_numpy(golden["emb_ids"])
    for tag in ("f32", "bf16"):
        G = as_dtype(golden[f"emb_{tag}_G"], tag)
        M = o.embedding_dot(ids.cuda(), G.cuda(), 3, 11)
        grad = o.embedding_wgrad(ids.cuda(), G.cuda(), 5, 11, 8.0, 5.0)
        after()
        assert O.rel_fro(M.sum(0), torch.from_numpy(golden[f"emb_{tag}_nv3_w"])) < 2e-2
        assert np.array_equal(grad.cpu().float().numpy(), golden[f"emb_{tag}_train_grad"])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [
    # n_t, n_v, T, d, vocab, share of tokens that carry one and the same id
    (6, 3, 200, 64, 50, 0.6),        # validation chain of ~360 tokens, train bucket of ~720
    (64, 2, 48, 24, 48, None),       # position ids: every id 64 times in the train rows (> 32), twice in val
    (40, 2, 1024, 16, 1000, 0.9),    # a train bucket above 32768 tokens: sorted in place in global memory
    (5, 40, 64, 40, 30, 0.5)])       # many validation samples, feature size not a multiple of 16
def test_embedding_with_heavily_repeated_ids(case, dtype):
    """Padding-like batches: one id carried by most tokens.  The dot products go through the
    per-(id, validation sample) pre-summed rows, the train gradient through the big-bucket kernel,
    and the train gradient stays bit-identical to the CPU's sequential index_add_."""
    n_t, n_v, T, d, vocab, share = case
    N = n_t + n_v
    g = torch.Generator().manual_seed(31)
    if share is None:
        ids = torch.arange(T).repeat(N, 1)
    else:
        ids = torch.randint(0, vocab, (N, T), generator=g)
        ids[torch.rand(N, T, generator=g) < share] = 7
    G = (torch.randn(N, T, d, generator=g) / d ** 0.5).to(dtype)
    o = ops()
    M = o.embedding_dot(ids.cuda(), G.cuda(), n_v, vocab)
    grad = o.embedding_wgrad(ids.cuda(), G.cuda(), n_t, vocab, float(N), float(n_t))
    after()
    assert O.rel_fro(M, O.embedding_dot_exact(ids, G, n_v)) < (1e-5 if dtype == torch.float32 else 1e-4)
    ref = O.embedding_train_grad(ids, G * N, n_v, vocab, sequential=True)
    assert torch.equal(grad.cpu().float(), ref.float())


# one call for both results, at the feature counts where a lane's share of a row changes (256, 512, 768,
# 1024 and beyond, ragged), rows of one, 32, 33 and many tokens side by side, more hot ids than slots
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(3, 2, 40, 256, 9), (3, 2, 64, 264, 200), (2, 1, 70, 520, 33), (4, 3, 33, 768, 5),
                                  (2, 2, 50, 776, 64), (3, 1, 37, 1032, 12), (2, 3, 45, 37, 20), (1, 1, 1, 8, 1),
                                  (4, 2, 8000, 8, 300)])
def test_embedding_hook(case, dtype):
    n_t, n_v, T, d, vocab = case
    N = n_t + n_v
    g = torch.Generator().manual_seed(41)
    ids = (torch.rand(N, T, generator=g).pow(2) * vocab).long().clamp_(max=vocab - 1)
    G = (torch.randn(N, T, d, generator=g) / d ** 0.5).to(dtype)
    M, grad = ops().embedding_hook(ids.cuda(), G.cuda(), n_v, vocab, float(N))
    after()
    assert O.rel_fro(M, O.embedding_dot_exact(ids, G, n_v)) < (1e-5 if dtype == torch.float32 else 1e-4)
    assert torch.equal(grad.cpu().float(), O.embedding_train_grad(ids, G * N, n_v, vocab, sequential=True).float())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab,n_v", [(9, 2), (1, 3), (9, 80)])       # joined rows, summed rows, many validation rows
def test_embedding_matrix_with_infinities(vocab, n_v, dtype):
    """Entries are infinite or NaN exactly where the plain sums are, and no other entry is touched."""
    n_t, T, d = 5, 40, 72
    N = n_t + n_v
    g = torch.Generator().manual_seed(12)
    ids = torch.randint(0, vocab, (N, T), generator=g)
    if n_v > 2:                  # an id of many validation tokens has a summed row, zero, for a sample without it
        ids[:, 10:10 + vocab] = torch.arange(vocab)
    G = (0.5 + torch.rand(N, T, d, generator=g)).to(dtype)
    G[1, 3, 5] = float("inf")
    G[2, 0, 0], G[2, 1, 1] = float("inf"), -float("inf")
    G[n_t + 1, 7, 9] = -float("inf")
    if dtype == torch.float32:
        G[3, 2, 2] = 3.4e38                      # finite, but beyond what a bf16 part can hold
        G[n_t:, :, 2] = 1e-3
    M = ops().embedding_dot(ids.cuda(), G.cuda(), n_v, vocab).cpu()
    after()
    R = torch.zeros(N, vocab, d, dtype=torch.float64)
    for i in range(N):
        R[i].index_add_(0, ids[i], G[i].double())
    # rows without the id are absent, not zero: they meet no infinity
    has = torch.zeros(N, vocab, dtype=torch.bool).scatter_(1, ids, True)
    want = torch.zeros(n_v, n_t, dtype=torch.float64)
    for v in range(n_v):
        for b in range(n_t):
            both = has[n_t + v] & has[b]
            want[v, b] = (R[n_t + v][both] * R[b][both]).sum()
    assert torch.equal(M.isnan(), want.isnan())
    assert torch.equal(M.isposinf(), want.isposinf()) and torch.equal(M.isneginf(), want.isneginf())
    fin = want.isfinite()
    assert ((M.double() - want)[fin].abs() <= 1e-5 * want[fin].abs()).all()


def test_embedding_out_of_range_ids_are_reported():
    """An id outside the table makes the reference's index_add_ raise.  The kernels skip such a token
    and record it; the next poll of the error word raises IndexError."""
    from ghostsuite_b200 import _lib
    n_t, n_v, T, d, vocab = 4, 2, 9, 16, 30
    g = torch.Generator().manual_seed(2)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=g)
    G = torch.randn(n_t + n_v, T, d, generator=g)
    good_M = ops().embedding_dot(ids.cuda(), G.cuda(), n_v, vocab)
    after()                                                   # nothing recorded for valid ids
    for row, col in ((1, 3), (n_t, 4)):                       # a train token, then a validation token
        bad = ids.clone()
        bad[row, col] = vocab
        M = ops().embedding_dot(bad.cuda(), G.cuda(), n_v, vocab)
        torch.cuda.synchronize()
        with pytest.raises(IndexError):
            _lib.poll_kernel_error()
        keep = torch.ones(n_t + n_v, T, 1)
        keep[row, col] = 0
        assert O.rel_fro(M, O.embedding_dot_exact(ids, G * keep, n_v)) < 1e-5
    bad = ids.clone()
    bad[0, 0] = -1
    ops().embedding_wgrad(bad.cuda(), G.cuda(), n_t, vocab, 1.0, float(n_t))
    torch.cuda.synchronize()
    with pytest.raises(IndexError):
        _lib.poll_kernel_error()
    _lib.poll_kernel_error()
    assert torch.isfinite(good_M).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(8, 6, 16, 24, 4, 6), (4, 130, 72, 200, 32, 32), (2, 300, 512, 136, 64, 64),
                                  (3, 1, 10, 20, 5, 3), (2, 257, 128, 256, 120, 34)])
def test_gradproj_dense(case, dtype):
    B, T, n_i, n_o, k_i, k_o = case
    A, G = make(B, T, n_i, n_o, dtype, seed=9)
    g = torch.Generator().manual_seed(10)
    P_i = torch.randn(k_i, n_i, generator=g) / k_i ** 0.5
    P_o = torch.randn(k_o, n_o, generator=g) / k_o ** 0.5
    o = ops()
    split = dtype == torch.float32
    Pr = o.prepare_projection(P_o.cuda(), split)
    Pc = o.prepare_projection(P_i.cuda(), split)
    total = k_o * k_i + 7
    buf = torch.full((B, total), 123.0, device="cuda")
    o.gradproj_dense(G.cuda(), A.cuda(), Pr, Pc, k_o, k_i, float(B), buf[:, 3:3 + k_o * k_i])
    after()
    ref = O.gradproj_dense(A, G, P_i, P_o, compute_dtype=torch.float64)
    got = buf[:, 3:3 + k_o * k_i].reshape(B, k_o, k_i)
    assert O.rel_fro(got, ref) < (1e-4 if split else 2e-2)
    # neighbours of the slice are untouched
    assert torch.all(buf[:, :3] == 123.0) and torch.all(buf[:, 3 + k_o * k_i:] == 123.0)


def test_gradproj_golden(golden):
    A = torch.from_numpy(golden["lin_f32_A"])
    G = torch.from_numpy(golden["lin_f32_G"])
    o = ops()
    P_i, P_o = torch.from_numpy(golden["gp_P_i"]), torch.from_numpy(golden["gp_P_o"])
    out = torch.empty(8, 24, device="cuda")
    o.gradproj_dense(G.cuda(), A.cuda(), o.prepare_projection(P_o.cuda(), True),
                     o.prepare_projection(P_i.cuda(), True), 6, 4, 8.0, out)
    after()
    assert O.rel_fro(out.reshape(8, 6, 4), torch.from_numpy(golden["gp_linear"])) < 1e-4
    assert torch.allclose(out.cpu().reshape(8, 6, 4), torch.from_numpy(golden["gp_linear"]), rtol=1e-3, atol=1e-4)
    # Conv1D: the out-grad is projected with P_i, the activations with P_o -> [k_i, k_o]
    P_i, P_o = torch.from_numpy(golden["gp_c1d_P_i"]), torch.from_numpy(golden["gp_c1d_P_o"])
    o.gradproj_dense(G.cuda(), A.cuda(), o.prepare_projection(P_i.cuda(), True),
                     o.prepare_projection(P_o.cuda(), True), 4, 6, 8.0, out)
    after()
    assert O.rel_fro(out.reshape(8, 4, 6), torch.from_numpy(golden["gp_c1d"])) < 1e-4
    assert torch.allclose(out.cpu().reshape(8, 4, 6), torch.from_numpy(golden["gp_c1d"]), rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [
    # B, T, d, vocab, k_i, k_o
    (3, 7, 12, 19, 5, 4),          # the golden case's sizes: everything smaller than one tile
    (4, 130, 72, 300, 32, 32),     # T straddles the 64-token blocks, d not a multiple of 16
    (2, 300, 512, 50, 64, 64),     # heavy id repetition, the largest single-launch block
    (3, 1, 10, 20, 3, 5),          # one token per sample, d with a 2-element tail
    (2, 65, 11, 40, 7, 9),         # odd feature size: the element-wise load path
    (2, 257, 128, 1000, 12, 85),   # k_o > 64: covered block by block
    (2, 33, 64, 64, 70, 66)])      # both larger than 64
def test_gradproj_embedding(case, dtype):
    B, T, d, vocab, k_i, k_o = case
    g = torch.Generator().manual_seed(21)
    ids = torch.randint(0, vocab, (B, T), generator=g)
    G = (torch.randn(B, T, d, generator=g) / d ** 0.5).to(dtype)
    P_i = torch.randn(k_i, vocab, generator=g) / k_i ** 0.5
    P_o = torch.randn(k_o, d, generator=g) / k_o ** 0.5
    o = ops()
    split = dtype == torch.float32
    Po = o.prepare_projection(P_o.cuda(), split)
    PiT = o.prepare_embedding_projection(P_i.cuda())
    total = k_o * k_i + 9
    buf = torch.full((B, total), 55.0, device="cuda")
    o.gradproj_embedding(ids.cuda(), G.cuda(), Po, PiT, k_o, k_i, 1.0, buf[:, 4:4 + k_o * k_i])
    after()
    ref = O.gradproj_embedding(ids, G, P_i, P_o, compute_dtype=torch.float64)
    got = buf[:, 4:4 + k_o * k_i].reshape(B, k_o, k_i)
    assert O.rel_fro(got, ref) < (1e-4 if split else 2e-2)
    assert torch.all(buf[:, :4] == 55.0) and torch.all(buf[:, 4 + k_o * k_i:] == 55.0)
    # a second call into the same buffer overwrites (the kernel adds into a block it zeroed itself)
    o.gradproj_embedding(ids.cuda(), G.cuda(), Po, PiT, k_o, k_i, 2.0, buf[:, 4:4 + k_o * k_i])
    after()
    assert O.rel_fro(buf[:, 4:4 + k_o * k_i].reshape(B, k_o, k_i), 2 * ref) < (1e-4 if split else 2e-2)


def test_gradproj_embedding_golden_and_bad_ids(golden):
    """The reference's per-token loop (golden output), then an id outside the table: the kernel skips
    it and the next poll raises IndexError, as indexing P_i[:, id] does in the reference."""
    ids = torch.from_numpy(golden["gp_emb_ids"])
    G = torch.from_numpy(golden["gp_emb_G"])
    P_i, P_o = torch.from_numpy(golden["gp_emb_P_i"]), torch.from_numpy(golden["gp_emb_P_o"])
    o = ops()
    Po = o.prepare_projection(P_o.cuda(), True)
    PiT = o.prepare_embedding_projection(P_i.cuda())
    out = o.gradproj_embedding(ids.cuda(), G.cuda(), Po, PiT, 4, 5)
    after()
    want = torch.from_numpy(golden["gp_emb"])
    assert O.rel_fro(out.reshape(3, 4, 5), want) < 1e-4
    assert torch.allclose(out.cpu().reshape(3, 4, 5), want, rtol=1e-3, atol=1e-4)
    bad = ids.clone()
    bad[1, 2] = 19                                        # vocab is 19
    out2 = o.gradproj_embedding(bad.cuda(), G.cuda(), Po, PiT, 4, 5)
    torch.cuda.synchronize()
    from ghostsuite_b200 import _lib
    with pytest.raises(IndexError):
        _lib.poll_kernel_error()
    _lib.poll_kernel_error()                              # the word was cleared
    keep = torch.ones(3, 7, dtype=torch.bool)
    keep[1, 2] = False
    ref = O.gradproj_embedding(ids, G * keep.unsqueeze(-1), P_i, P_o, compute_dtype=torch.float64)
    assert O.rel_fro(out2.reshape(3, 4, 5), ref) < 1e-4     # the bad token contributed nothing


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(3, 5, 64), (16, 16, 98304), (8, 40, 1000), (33, 17, 4096),
                                  (5, 3, 12345), (1, 1, 7), (16, 8, 917504)])
def test_projection_similarity(case, dtype):
    n1, n2, D = case
    g = torch.Generator().manual_seed(22)
    P1 = torch.randn(n1, D, generator=g).to(dtype)
    P2 = (torch.randn(n2, D, generator=g) + 0.05 * torch.randn(1, D, generator=g)).to(dtype)
    S = ops().projection_similarity(P1.cuda(), P2.cuda(), 0.5)
    after()
    ref = 0.5 * O.projection_similarity(P1, P2)
    assert S.shape == (n1, n2) and S.dtype == torch.float32
    assert O.rel_fro(S, ref) < 1e-4
    # rows of a wider buffer (the engine's [B, total_proj_dim] buffer, a column range of it)
    if D >= 64:
        wide = torch.zeros(n1, D + 24, dtype=dtype, device="cuda")
        wide[:, 8:8 + D] = P1.cuda()
        S2 = ops().projection_similarity(wide[:, 8:8 + D], P2.cuda(), 0.5)
        after()
        assert O.rel_fro(S2, ref) < 1e-4


# every block shape of the kernel with ragged edges, odd and tiny contraction lengths
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(16, 8, 40), (15, 16, 1000), (3, 70, 264), (31, 25, 2048), (70, 9, 33), (65, 130, 8200), (1, 1, 1)])
def test_projection_similarity_block_shapes(case, dtype):
    n1, n2, D = case
    g = torch.Generator().manual_seed(23)
    a, b = (torch.randn(n, D, generator=g).to(dtype) for n in (n1, n2))
    S = ops().projection_similarity(a.cuda(), b.cuda(), 0.5)
    after()
    # float32 rows carry two bf16 parts each: 2^-16 per product, relative to the row norms
    err = (S.cpu().double() - 0.5 * a.double() @ b.double().t()).abs()
    assert (err <= 2.0 ** -15 * a.double().norm(dim=1)[:, None] * b.double().norm(dim=1)[None]).all()


# more rows than ops.SIMILARITY_KERNEL_MAX_ROWS: bf16 sets go to the kernel, also as columns of wider rows; gradients, overlapping
# rows and mixed types stay where they were
@pytest.mark.parametrize("n1, n2, D", [(2, 129, 96), (129, 3, 257), (512, 200, 128), (700, 513, 200), (513, 2, 101), (1, 129, 1), (1, 200, 512), (513, 2, 31)])
def test_projection_similarity_of_large_bf16_sets(n1, n2, D):
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    g = torch.Generator(device="cuda").manual_seed(25)
    a, b = (torch.randn(n, D, generator=g, device="cuda").bfloat16() for n in (n1, n2))
    wide = torch.full((n1, D + 3), 1e30, device="cuda").bfloat16()
    wide[:, 2:2 + D] = a
    ref = a.double() @ b.double().t()
    # exact products; the sums of 2 D / 32 partial sums are off by 2^-24 each at most, those inside a step by one truncation per product
    bound = (D + 32) * 2.0 ** -23 * a.double().abs() @ b.double().abs().t()
    before = ops().launch_count()
    for rows in (a, wide[:, 2:2 + D]):
        S = U.projection_similarity(rows, b)
        after()
        assert S.dtype == torch.float32 and ((S.double() - ref).abs() <= bound).all()
    # short rows and many unaligned ones stay with the GEMM
    kernel = D >= 96 and (D % 8 == 0 or max(n1, n2) <= 512)
    assert ops().launch_count() > before if kernel else ops().launch_count() == before
    bits = a.clone()
    bits[0, 0] = float("inf")
    assert torch.equal(torch.isfinite(U.projection_similarity(bits, b)), torch.isfinite(bits.double() @ b.double().t()))
    count = ops().launch_count()
    assert U.projection_similarity(a.clone().requires_grad_(), b).grad_fn is not None
    assert U.projection_similarity(a[:1].expand(max(n1, 200), D), b).shape == (max(n1, 200), n2)
    assert U.projection_similarity(a, b.float()).dtype == torch.float32
    assert ops().launch_count() == count


# no less exact than the float32 product they had before; the two round in different orders, so that their errors, of 258 scores and more,
# differ by a few percent where neither is the better one
@pytest.mark.parametrize("n1, n2, D", [(1, 200, 512), (1, 200, 65536), (2, 129, 96), (200, 3, 64), (3, 200, 1000), (16, 512, 4096), (200, 2, 65536)])
def test_error_of_large_bf16_similarity_sets(n1, n2, D):
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    g = torch.Generator(device="cuda").manual_seed(26)
    errors = []
    for _ in range(4):
        a, b = (torch.randn(n, D, generator=g, device="cuda").bfloat16() for n in (n1, n2))
        ref = a.double() @ b.double().t()
        errors.append([((x.double() - ref).norm() / ref.norm()).item() ** 2 for x in (U.projection_similarity(a, b), a.float() @ b.float().t())])
    after()
    assert sum(e[0] for e in errors) <= 1.1 ** 2 * sum(e[1] for e in errors)


# one row against more than 128: rows that no four of a warp fill, one warp to 64 of them to a row, one round of loads and several, columns that end
# inside one; rows on 16-byte boundaries and anywhere, between values that nothing may take in; scores as a row, a column, and a column of
# wider rows
@pytest.mark.parametrize("n, D", [(129, 96), (130, 97), (131, 264), (132, 511), (133, 4104), (200, 2049), (129, 131080), (130, 70001), (9475, 256), (9480, 101)])
def test_similarity_of_one_bf16_row(n, D):
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(27)
    nan = torch.full((n * (D + 8) + 16,), float("nan"), device="cuda").bfloat16()
    for offset in (0, 8) if D % 8 == 0 else (0, 3):
        one = nan[:D + 16].clone()[offset:offset + D]
        many = nan.clone()[offset:offset + n * (D + 8)].view(n, D + 8)[:, :D]
        one.copy_(torch.randn(D, generator=g, device="cuda"))
        many.copy_(torch.randn(n, D, generator=g, device="cuda"))
        ref = 0.5 * (many.double() @ one.double())
        # products are exact; a lane's chains are D / 256 sums, then a tree over elements, lanes, warps and CTAs
        bound = (D / 256 + 16) * 2.0 ** -24 * 0.5 * (many.double().abs() @ one.double().abs())
        one = one.view(1, D)
        rows = [ops().projection_similarity(one, many, 0.5), ops().projection_similarity(many, one, 0.5).t()]
        wide = torch.full((n, 3), 7.0, device="cuda")
        _lib.check(lib.ghost_projection_similarity(many.data_ptr(), one.data_ptr(), 0, n, 1, D, D + 8, D, 0.5, wide.data_ptr(), 3, torch.cuda.current_stream().cuda_stream))
        after()
        for S in (*rows, wide[:, :1].t()):
            assert ((S[0].double() - ref).abs() <= bound).all()
        assert torch.equal(rows[0], rows[1]) and torch.equal(rows[0], wide[:, :1].t()) and (wide[:, 1:] == 7).all()
        assert torch.equal(rows[0], ops().projection_similarity(one, many, 0.5))           # the same bits again


# one stage, one cluster and many of them; rows that TMA reads and rows that it cannot (odd lengths, odd pitches), each at
# the ends of a panel of 32 floats / 64 bf16 elements; scores with and without whole 16-byte pieces per row
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [8, 31, 256, 257, 2055, 4096, 65536 + 24, 65536 + 25])
@pytest.mark.parametrize("n", [(2, 3), (18, 74), (40, 33), (64, 64)])
def test_projection_similarity_splits_and_pitches(n, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(24)
    a, b = (torch.randn(k, D, generator=g, device="cuda").to(dtype) for k in n)
    wide = torch.full((n[0], D + 3), 1e30, device="cuda").to(dtype)
    wide[:, 2:2 + D] = a
    ref = a.double() @ b.double().t()
    bound = 2.0 ** -15 * a.double().norm(dim=1)[:, None] * b.double().norm(dim=1)[None]
    for rows in (a, wide[:, 2:2 + D]):
        S = ops().projection_similarity(rows, b)
        after()
        assert ((S.double() - ref).abs() <= bound).all()



def test_small_reduce_batch_matches_single_launches():
    """One batched launch for many layers' small reductions against the per-layer kernels: more jobs
    than fit one launch, mixed sizes, Gram only / sum only / both, bf16 and fp32 sums."""
    o = ops()
    g = torch.Generator().manual_seed(23)
    jobs, want = [], []
    for i in range(110):
        n_t, n_v = (5, 3) if i % 3 else (32, 8)
        F = (768, 10, 3072, 37, 1)[i % 5]
        X = torch.randn(n_t + n_v, F, generator=g).cuda()
        job = {"X": X, "n_train": n_t, "n_val": n_v}
        rec = {}
        if i % 4 != 1:
            job["M"] = torch.full((n_v, n_t), 7.0, device="cuda")
            job["dot_scale"] = 0.5
            rec["M"] = o.small_gram(X, n_v, 0.5)
        if i % 4 != 2:
            dt = torch.bfloat16 if i % 2 else torch.float32
            job["sum_out"] = torch.full((F,), 7.0, dtype=dt, device="cuda")
            job["sum_scale"] = 0.25
            rec["sum"] = o.rows_sum(X, n_t, 0.25, dt)
        jobs.append(job)
        want.append(rec)
    from ghostsuite_b200 import _lib
    l0 = _lib.launch_count()
    o.small_reduce_batch(jobs)
    assert _lib.launch_count() - l0 == 3                      # 48 jobs per launch
    after()
    for job, rec in zip(jobs, want):
        if "M" in rec:
            assert torch.equal(job["M"], rec["M"])
        if "sum" in rec:
            assert torch.equal(job["sum_out"], rec["sum"])


# validation rows on both sides of a block's 8 and 16, train rows of one block and of two, vectors staged in one round and in more
@pytest.mark.parametrize("n_t,n_v", [(32, 9), (5, 16), (40, 17), (33, 35)])
@pytest.mark.parametrize("F", [37, 1024, 4100])
def test_pass_reduce_of_many_validation_rows(n_t, n_v, F):
    o = ops()
    X = torch.randn(n_t + n_v, F, generator=torch.Generator().manual_seed(5)).cuda()
    M, S = torch.full((n_v, n_t), 7.0, device="cuda"), torch.full((F,), 7.0, device="cuda")
    few = torch.full((3, n_t), 7.0, device="cuda")
    vec, = o.pass_reduce([{"X": X, "n_train": n_t, "n_val": n_v, "M": M, "sum_out": S, "dot_scale": 0.5},
                          {"X": X, "n_train": n_t, "n_val": 3, "M": few, "dot_scale": 0.5}], [M])
    after()
    T, V = X[:n_t].double(), X[n_t:].double()
    # chains of F / 256 products in each of 256 accumulators, then pairs: a rounding of 2^-24 per level
    bound = (F / 256 + 10) * 2.0 ** -24 * 0.5 * (V.abs() @ T.abs().t())
    assert ((M.double() - 0.5 * V @ T.t()).abs() <= bound).all()
    assert torch.equal(few, M[:3])
    assert ((vec.double() - M.double().sum(0)).abs() <= (n_v / 8 + 3) * 2.0 ** -24 * M.double().abs().sum(0)).all()
    assert ((S.double() - T.sum(0)).abs() <= n_t * 2.0 ** -24 * T.abs().sum(0)).all()


# fewer rows than a block has lanes, behind a launch that left NaN in the shared memory of every SM; a share of columns in one round and two
@pytest.mark.parametrize("n_t,n_v", [(1, 1), (3, 1), (31, 7), (33, 9)])
@pytest.mark.parametrize("F", [30, 8192, 8201])
def test_pass_reduce_reads_only_rows_that_exist(n_t, n_v, F):
    o = ops()
    X = torch.randn(n_t + n_v, F, generator=torch.Generator().manual_seed(6)).cuda()
    bad = torch.full((48, 8200), float("nan"), device="cuda")
    spoilt = [{"X": bad, "n_train": 32, "n_val": 16, "M": torch.empty(16, 32, device="cuda")} for _ in range(24)]
    o.pass_reduce(spoilt, [j["M"] for j in spoilt[:1]])
    M, S = torch.full((n_v, n_t), 7.0, device="cuda"), torch.full((F,), 7.0, device="cuda")
    vec, = o.pass_reduce([{"X": X, "n_train": n_t, "n_val": n_v, "M": M, "sum_out": S}], [M])
    after()
    T, V = X[:n_t].double(), X[n_t:].double()
    bound = (F / 256 + 10) * 2.0 ** -24 * (V.abs() @ T.abs().t())        # as above
    assert ((M.double() - V @ T.t()).abs() <= bound).all()
    assert ((vec.double() - M.double().sum(0)).abs() <= (n_v / 8 + 3) * 2.0 ** -24 * M.double().abs().sum(0)).all()
    assert ((S.double() - T.sum(0)).abs() <= n_t * 2.0 ** -24 * T.abs().sum(0)).all()


# one matrix on its own, beyond what the batched launch's blocks take: vector and scalar loads, remainders
@pytest.mark.parametrize("n_t,n_v,F", [(300, 30, 772), (2000, 3, 1001), (70, 40, 4100), (5, 3, 150001), (600, 8, 512)])
def test_small_gram_of_large_vectors(n_t, n_v, F):
    X = torch.randn(n_t + n_v, F, generator=torch.Generator().manual_seed(3)).cuda()
    M = ops().small_gram(X, n_v, 0.5)
    after()
    want = 0.5 * X[n_t:].double() @ X[:n_t].double().t()
    # 256 float32 accumulators of F / 256 products each, then pairs: a rounding of 2^-24 per level of the sum
    bound = (F / 256 + 9) * 2.0 ** -24 * 0.5 * (X[n_t:].double().abs() @ X[:n_t].double().abs().t())
    assert ((M.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("n,F", [(4, 20003), (33, 50257), (300, 100), (9, 1), (7, 18944), (1, 31)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_sum_gives_the_batched_launchs_bits(n, F, dtype):
    o = ops()
    X = torch.randn(n, F, generator=torch.Generator().manual_seed(4)).cuda()
    S = torch.empty(F, dtype=dtype, device="cuda")
    o.small_reduce_batch([{"X": X, "n_train": n, "n_val": 0, "sum_out": S, "sum_scale": 0.25}])
    got = o.rows_sum(X, n, 0.25, dtype)
    after()
    assert torch.equal(got, S)
    more = o.rows_sum(X, n, 0.25, dtype, out=got.clone(), accumulate=True)
    after()
    assert O.rel_fro(more, 2 * S.double()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22)


def test_more_train_samples_than_a_grid_has_blocks():
    """Jobs of more than 32 x 65535 train samples: the blocks take several groups of 32 in turn."""
    o = ops()
    n_t = 32 * 65535 + 70
    X = torch.randint(-4, 5, (n_t + 3, 1), generator=torch.Generator().manual_seed(1)).float().cuda()
    M, S = torch.empty(3, n_t, device="cuda"), torch.empty(1, device="cuda")
    o.small_reduce_batch([{"X": X, "n_train": n_t, "n_val": 3, "M": M, "sum_out": S}])
    vec, again = o.pass_reduce([{"X": X, "n_train": n_t, "n_val": 3, "M": (M2 := torch.empty_like(M))}], [M2, M])
    rows = o.rows_sum(X, n_t, 1.0, torch.float32)
    after()
    want = X[n_t:] * X[:n_t].T                       # whole numbers: exact
    assert torch.equal(M, want) and torch.equal(M2, want)
    assert torch.equal(vec, want.sum(0)) and torch.equal(again, want.sum(0))
    assert S.item() == rows.item() == X[:n_t].sum().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("any_path,use_gram", [(True, True), (False, True), (False, False)])
def test_dense_hook_with_separate_column_sums(any_path, use_gram, dtype):
    from ghostsuite_b200 import _lib
    A, G = make(7, 5, 40, 24, dtype)
    res, launches = [], []
    for fuse in (True, False):
        l0 = _lib.launch_count()
        res.append(ops().dense_hook(A.cuda(), G.cuda(), 2, False, use_gram, dtype, 1.0, True, dtype, any_path, fuse))
        launches.append(_lib.launch_count() - l0)
    after()
    # the per-sample path adds a handful of blocks' sums in any order: a rounding of 2^-24 each
    assert O.rel_fro(res[0][0], res[1][0].double()) < 8 * 2.0 ** -24 and torch.equal(res[0][1], res[1][1])
    for r in res:
        assert O.rel_fro(r[2], G.double().sum(1)) < 1e-6
    taken_along = any_path or (not use_gram and dtype == torch.bfloat16)
    assert launches[1] - launches[0] == (1 if taken_along else 0)


def test_result_buffers_and_samples_are_checked_before_anything_is_written():
    o = ops()
    X = torch.randn(1, 8, 16).cuda()
    good = torch.zeros(16, 16).cuda()
    for out in (torch.zeros(16, 15).cuda(), torch.zeros(16, 32).cuda()[:, :16], good.t()[:8]):
        with pytest.raises(ValueError):
            o.wgrad(X, X, 1.0, torch.float32, out=out)
    assert torch.equal(o.wgrad(X, X, 1.0, torch.float32, out=good.view(256)).view(16, 16), o.wgrad(X, X, 1.0, torch.float32))
    ids, G = torch.zeros(3, 4, dtype=torch.long).cuda(), torch.randn(3, 4, 8).cuda()
    for kw in (dict(n_train=4), dict(vocab=6, out=torch.zeros(5, 8).cuda()), dict(ids=ids[:, :3]), dict(ids=ids[:1])):
        args = dict(ids=ids, G=G, n_train=2, vocab=5, pre_scale=1.0, divisor=2.0)
        args.update(kw)
        with pytest.raises(ValueError):
            o.embedding_wgrad(**args)
    after()


def test_matrix_listed_twice_beside_the_job_that_fills_it():
    X = torch.randn(37, 96, generator=torch.Generator().manual_seed(2)).cuda()
    M, other = torch.empty(5, 32, device="cuda"), torch.randn(5, 32).cuda()
    first, between, second = ops().pass_reduce([{"X": X, "n_train": 32, "n_val": 5, "M": M}], [M, other, M])
    after()
    assert torch.equal(first, second) and O.rel_fro(first, M.double().sum(0)) < 1e-6
    assert O.rel_fro(between, other.double().sum(0)) < 1e-6


def test_conv_tokens_refuses_what_its_grid_cannot_hold():
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    src, dst = torch.zeros(64, device="cuda"), torch.zeros(64, dtype=torch.bfloat16, device="cuda")
    for cols, cpad in ((64 * 65535 + 8, 64 * 65535 + 8), (8, 64 * 65535 + 8)):
        rc = lib.ghost_conv_tokens_bf16(src.data_ptr(), 1, 1, cols, 1, 1, 1, 1, 1, 1, 0, 0, 1, 1, dst.data_ptr(), cpad, cpad, 1,
                                        0, 0, 0, 0, torch.cuda.current_stream().cuda_stream)
        assert rc == _lib.GHOST_ERR_INVALID
    after()


def test_error_codes_are_python_exceptions():
    o = ops()
    A = torch.randn(4, 3, 8, device="cuda")
    with pytest.raises(ValueError):
        o.gram_dot(A, A, 4)            # no training samples
    with pytest.raises(ValueError):
        o.small_gram(A.reshape(4, 24), 4)
    with pytest.raises(RuntimeError):
        o.colsum(A.cpu())
    # the two-pass entry points through the raw C ABI: every refusal is GHOST_ERR_INVALID with a message
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    X = torch.zeros(6, 16, 64, dtype=torch.bfloat16, device="cuda")
    tiles = torch.zeros(6 * 32768, dtype=torch.bfloat16, device="cuda")
    M = torch.zeros(64, device="cuda")
    nbytes = lib.ghost_persample_tiles_bytes(6, 64, 64)
    assert nbytes == 6 * 65536 and lib.ghost_persample_tiles_bytes(0, 64, 64) == 0
    args = lambda s0, ns, nb: (X.data_ptr(), X.data_ptr(), 6, 16, 64, 64, 64, 64, s0, ns, 0, None, tiles.data_ptr(), nb, None)
    assert lib.ghost_persample_tiles_bf16(*args(0, 6, nbytes)) == 0
    assert lib.ghost_persample_tiles_bf16(*args(4, 3, nbytes)) == -1 and b"sample range" in lib.ghost_last_error()
    assert lib.ghost_persample_tiles_bf16(*args(0, 6, nbytes - 1)) == -1 and b"too small" in lib.ghost_last_error()
    dot = lambda ranks, per, n_t, grad: lib.ghost_tile_dot_bf16(tiles.data_ptr(), ranks, per, tiles.data_ptr(), n_t, 64, 64, 1.0,
                                                                M.data_ptr(), grad, 0, 1.0, 0, None)
    assert dot(1, 2, 4, None) == 0
    assert dot(4, 3, 4, None) == -1 and b"per rank" in lib.ghost_last_error()
    assert dot(1, 2, 33, tiles.data_ptr()) == -1 and b"32 train samples" in lib.ghost_last_error()
    assert dot(1, 2, 0, None) == -1
    after()


# ------------------------------------------------------------------------------------------------
# benchmark model helper: fused token cross-entropy against torch's own
# ------------------------------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(37, 1000, 1000), (64, 50304, 50257), (5, 72, 61)])
def test_fused_token_loss_matches_torch(shape, dtype):
    from ghostsuite_b200.workloads import _FusedTokenLoss
    rows, cols, valid = shape
    g = torch.Generator().manual_seed(5)
    logits = (torch.randn(rows, cols, generator=g) * 3).to(dtype).cuda().requires_grad_(True)
    target = torch.randint(0, valid, (rows,), generator=g)
    target[::7] = -100
    target = target.cuda()
    loss = _FusedTokenLoss.apply(logits, target, valid)
    (loss * 1.7).backward()
    ref_logits = logits.detach().float().clone().requires_grad_(True)
    masked = ref_logits[:, :valid]
    ref = torch.nn.functional.cross_entropy(masked, target, ignore_index=-100)
    (ref * 1.7).backward()
    assert abs(loss.item() - ref.item()) <= 2e-5 * max(1.0, abs(ref.item()))
    got = logits.grad.float()
    want = ref_logits.grad
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5       # relative Frobenius; bf16 = one rounding of the result
    assert (got - want).norm() <= tol * want.norm()
    assert torch.count_nonzero(got[:, valid:]) == 0
    assert torch.count_nonzero(got[::7]) == 0
    # a retained graph backpropagated twice with different upstream gradients
    x2 = logits.detach().clone().requires_grad_(True)
    loss2 = _FusedTokenLoss.apply(x2, target, valid)
    loss2.backward(retain_graph=True)
    g1 = x2.grad.float().clone()
    x2.grad = None
    (loss2 * 0.25).backward()
    assert (g1 * 1.7 - want).norm() <= tol * want.norm()
    assert (x2.grad.float() * 4 * 1.7 - want).norm() <= tol * want.norm()
    # logits that need no gradient take the forward-only kernel
    assert abs(_FusedTokenLoss.apply(logits.detach(), target, valid).item() - ref.item()) <= 2e-5 * max(1.0, abs(ref.item()))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(6, 5, 64), (9, 33, 768), (3, 17, 4096), (4, 7, 30)])
def test_rmsnorm_persample(shape, dtype):
    N, T, F = shape
    g = torch.Generator().manual_seed(21)
    A = (torch.randn(N, T, F, generator=g) * 2 + 0.3).to(dtype)
    G = torch.randn(N, T, F, generator=g).to(dtype)
    gw, gsum = ops().layernorm_persample(A.cuda(), G.cuda(), 1e-6, rms=True)
    want = O.rmsnorm_persample_exact(A, G, 1e-6)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert O.rel_fro(gw, want) < tol
    assert O.rel_fro(gsum, G.double().sum(1)) < tol


# ids with 1 to 40 train and up to 4 validation tokens: load batches, sort sizes, the line between short and long
# rows, several join items an id; divisors on and off a power of two
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n_t,n_v,d", [(8, 3, 8), (8, 2, 264), (6, 3, 768), (1, 1, 520), (16, 4, 1024), (5, 2, 37)])
def test_embedding_hook_small_rows_exact(dtype, n_t, n_v, d):
    """Whole numbers up to 3: the matrix and the sums are exact in any order, the gradient is two roundings."""
    gen = torch.Generator().manual_seed(d + n_t)
    train = [k for k in range(60) for _ in range(k % 41)]
    val = [k for k in range(60) for _ in range((k * 7) % 5)]
    T = max(-(-len(train) // n_t), -(-len(val) // n_v))
    train += [63] * (n_t * T - len(train))             # an id of the train tokens only
    val += [62] * (n_v * T - len(val))                 # and one of the validation tokens only
    ids = torch.cat([torch.tensor(train)[torch.randperm(n_t * T, generator=gen)].view(n_t, T),
                     torch.tensor(val)[torch.randperm(n_v * T, generator=gen)].view(n_v, T)])
    G = torch.randint(-3, 4, (n_t + n_v, T, d), generator=gen).to(dtype)
    M, grad = ops().embedding_hook(ids.cuda(), G.cuda(), n_v, 64, 1.0)
    after()
    per = torch.zeros(n_t + n_v, 64, d, dtype=torch.float64)
    per.scatter_add_(1, ids.unsqueeze(-1).expand(-1, -1, d), G.double())
    assert torch.equal(M.cpu().double(), per[n_t:].flatten(1) @ per[:n_t].flatten(1).T)
    assert torch.equal(grad.cpu(), (per[:n_t].sum(0).to(dtype) / n_t).to(dtype))


# tokens around what one cluster buckets (4096, 8192) and around a warp; the table larger and smaller than them, ids of one side
# only, ids that most tokens share, ids outside of the table
@pytest.mark.parametrize("n_t,n_v,T,vocab", [(1, 1, 1, 1), (3, 2, 13, 5), (7, 1, 1024, 300), (6, 2, 1024, 50000), (3, 1, 2048, 7),
                                             (2731, 1, 3, 900), (4, 4, 1023, 20001), (1, 5, 700, 64), (3, 1, 1024, 9000), (16, 1, 241, 77)])
def test_embedding_buckets_of_one_cluster(n_t, n_v, T, vocab):
    from ghostsuite_b200 import _lib
    gen = torch.Generator().manual_seed(T)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=gen)
    common = torch.rand(ids.shape, generator=gen)
    ids[common < 0.3] = 0
    ids[:n_t][common[:n_t] > 0.95] = vocab // 2          # mostly train tokens
    G = torch.randint(-3, 4, (n_t + n_v, T, 8), generator=gen).float()
    bad = ids.clone()
    bad[common > 0.999] = vocab + 3
    for tokens in (ids, bad):
        keep = tokens < vocab
        M, grad = ops().embedding_hook(tokens.cuda(), G.cuda(), n_v, vocab, 1.0)
        torch.cuda.synchronize()
        if bool(keep.all()):
            _lib.poll_kernel_error()
        else:
            with pytest.raises(IndexError):
                _lib.poll_kernel_error()
        # whole numbers: exact in any order
        x, k = (G * keep.unsqueeze(-1)).double(), tokens.clamp(max=vocab - 1)
        val = torch.zeros(n_v, vocab, 8, dtype=torch.float64).scatter_add_(1, k[n_t:].unsqueeze(-1).expand(-1, -1, 8), x[n_t:])
        ref = torch.stack([(val[:, k[b]] * x[b]).sum((1, 2)) for b in range(n_t)], dim=1)
        gref = torch.zeros(vocab, 8, dtype=torch.float64).index_add_(0, k[:n_t].flatten(), x[:n_t].flatten(0, 1))
        assert torch.equal(M.cpu().double(), ref)
        assert torch.equal(grad.cpu(), (gref.float() / n_t))


# both sides of what one cluster clears: 4 MB of counts (0.75 without a matrix), 2 MB of sums above 2048 tokens; twice the tokens
# for both results only
@pytest.mark.parametrize("n_t,n_v,T,vocab,matrix,grad,one", [
    (9, 2, 2, 1048564, True, False, True), (9, 2, 2, 1048565, True, False, False),
    (9, 2, 2, 196596, False, True, True), (9, 2, 2, 196597, False, True, False), (9, 2, 2, 196597, True, True, True),
    (1024, 1024, 1, 70, True, False, True), (2000, 131, 1, 70, True, True, True), (2000, 132, 1, 70, True, True, False),
    (2000, 2000, 1, 70, True, False, False), (2500, 9, 2, 70, True, True, True), (1250, 1250, 2, 70, True, False, False),
    (2500, 9, 2, 70, False, True, False)])
def test_embedding_buckets_by_what_has_to_be_cleared(n_t, n_v, T, vocab, matrix, grad, one):
    from ghostsuite_b200 import _lib
    gen = torch.Generator().manual_seed(n_t)
    ids = torch.randint(0, min(vocab, 70), (n_t + n_v, T), generator=gen)
    ids[ids >= 35] += vocab - 70
    G = torch.randint(-3, 4, (n_t + n_v, T, 8), generator=gen).float()
    ids_d, G_d = ids.cuda(), G.cuda()
    before, M, out = _lib.launch_count(), None, None
    if matrix and grad:
        M, out = ops().embedding_hook(ids_d, G_d, n_v, vocab, 1.0)
    elif matrix:
        M = ops().embedding_dot(ids_d, G_d, n_v, vocab)
    else:
        out = ops().embedding_wgrad(ids_d[:n_t], G_d[:n_t], n_t, vocab, 1.0, n_t)
    # buckets; join, rounding of a matrix that shared memory does not hold; gradient
    assert _lib.launch_count() - before == (1 if one else 4) + (1 + (n_t * n_v > 4096) if matrix else 0) + grad
    after()
    small = torch.where(ids >= 35, ids - (vocab - 70), ids)
    hot = torch.nn.functional.one_hot(small, 70).double()
    rows = torch.einsum("nti,ntd->nid", hot, G.double())               # whole numbers: exact in any order
    if matrix:
        assert torch.equal(M.cpu().double(), rows[n_t:].flatten(1) @ rows[:n_t].flatten(1).t())
    if grad:
        ref = torch.zeros(vocab, 8).index_add_(0, ids[:n_t].flatten(), G[:n_t].flatten(0, 1)) / n_t
        assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("n_t,n_v,T", [(3, 2, 40), (5, 1, 1024)])
def test_embedding_dot_of_the_largest_table(n_t, n_v, T):
    """2^31 - 1 rows: the counts and the totals before them are more words than an int counts, and all of them are
    cleared, whatever the workspace (34 GB) held."""
    from ghostsuite_b200 import _lib
    lib, vocab, d = _lib.load(), 2 ** 31 - 1, 8
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, 60, (n_t + n_v, T), generator=g)
    ids[ids >= 30] += vocab - 60
    G = torch.randint(-3, 4, (n_t + n_v, T, d), generator=g).float()
    same = (ids[n_t:, None, :, None] == ids[None, :n_t, None, :]).double()
    ref = torch.einsum("vbst,vsd,btd->vb", same, G[n_t:].double(), G[:n_t].double())
    size = int(lib.ghost_embedding_pass_workspace_bytes(n_t, n_v, T, vocab, d))
    ws = torch.full((size,), 0x5b, dtype=torch.uint8, device="cuda")
    M, ids_d, G_d = torch.full((n_v, n_t), float("nan"), device="cuda"), ids.cuda(), G.cuda()
    _lib.check(lib.ghost_embedding_dot(ids_d.data_ptr(), G_d.data_ptr(), 1, n_t, n_v, T, d, vocab, 1.0, M.data_ptr(), ws.data_ptr(), size,
                                       torch.cuda.current_stream().cuda_stream))
    after()
    del ws
    torch.cuda.empty_cache()
    assert torch.equal(M.cpu().double(), ref)          # whole numbers: exact in any order


# widths around the lines of the block-per-rows kernel (1024, 2048, 4096, 8192, multiples of eight or not), row
# counts that leave a group of rows unfinished, one row, several splits
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,T,F", [(2, 1, 1032), (3, 5, 2048), (1, 387, 731), (2, 130, 4104), (2, 33, 8192), (1, 9, 8189),
                                   (2, 67, 1025), (3, 200, 2056), (1, 3, 8200), (5, 7, 3)])
def test_norm_wide_rows(dtype, rms, N, T, F):
    gen = torch.Generator().manual_seed(F)
    A = (torch.randn(N, T, F, generator=gen) * 1.5 + 0.3).to(dtype)
    G = (torch.randn(N, T, F, generator=gen) / F ** 0.5).to(dtype)
    gw, gb = ops().layernorm_persample(A.cuda(), G.cuda(), 1e-5, rms=rms)
    after()
    x, g = A.double(), G.double()
    x = x if rms else x - x.mean(-1, keepdim=True)
    x = x / (x.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()
    # float32 sums of F values and of T rows around values of order one: a few ulp of sqrt(F + T)
    assert O.rel_fro(gw, (g * x).sum(1)) < 2e-6
    assert O.rel_fro(gb, g.sum(1)) < 2e-6


# rows that begin anywhere, as many features a thread as the width needs (10, 12, 16 of 256 and of 512 threads), three or two rows at a
# time: widths on both sides of each form, row counts that leave a group unfinished, chains that end inside one
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,T,F", [(2, 1, 2049), (1, 37, 2559), (2, 100, 2561), (1, 5, 3071), (1, 34, 3073), (2, 70, 4097), (1, 101, 5119), (1, 4, 5121),
                                   (2, 35, 6143), (1, 7, 6145)])
def test_norm_rows_that_begin_anywhere(dtype, rms, N, T, F):
    test_norm_wide_rows(dtype, rms, N, T, F)


# rows of 16-byte pieces, 16 features for as many threads as the width needs: the widest and narrowest row of each form
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,T,F", [(2, 3, 2056), (1, 67, 3072), (2, 34, 3080), (1, 5, 4096), (2, 67, 4104), (1, 33, 5120), (1, 4, 5128), (2, 66, 6144),
                                   (1, 7, 6152), (1, 40, 7168), (1, 3, 7176)])
def test_norm_rows_of_pieces(dtype, rms, N, T, F):
    test_norm_wide_rows(dtype, rms, N, T, F)


# (B, T, columns of G, of A, k_r, k_c): one unit of 128 tokens to more than the GPU has SMs, so that every cluster size
# and none is met, with fewer stages of columns than CTAs among them; token counts around a unit; columns that no
# 16-byte load fits; ranks on both sides of each instantiation's largest
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(1, 1, 7, 5, 1, 1), (1, 10, 4407, 452, 44, 44), (2, 129, 333, 1000, 16, 17), (16, 127, 130, 70, 33, 9),
                                  (17, 128, 512, 300, 64, 64), (35, 100, 260, 516, 5, 60), (3, 300, 2050, 3072, 32, 48),
                                  (75, 64, 200, 136, 20, 20), (160, 33, 97, 104, 9, 4), (5, 140, 640, 259, 100, 128),
                                  (80, 200, 321, 192, 128, 65),
                                  # samples of several units in a cluster of eight, four, two, and too many for one
                                  (8, 1000, 64, 130, 7, 11), (3, 129, 72, 70, 64, 64), (32, 300, 100, 64, 17, 128), (33, 300, 64, 64, 5, 6),
                                  (72, 257, 66, 128, 20, 12), (7, 1025, 128, 64, 100, 128),
                                  # units shared by six CTAs (of 20 only with float32's longer chains, else four), four (24 units) and
                                  # three (38), whose tokens do not divide evenly
                                  (18, 128, 900, 1000, 40, 33), (20, 90, 2000, 64, 16, 16), (2, 1500, 1300, 700, 64, 64), (38, 128, 640, 520, 9, 64)])
def test_gradproj_dense_unit_counts_and_widths(case, dtype):
    B, T, n_r, n_c, k_r, k_c = case
    g = torch.Generator().manual_seed(17)
    G, A = torch.randn(B, T, n_r, generator=g).to(dtype), torch.randn(B, T, n_c, generator=g).to(dtype)
    P_r, P_c = torch.randn(k_r, n_r, generator=g) / k_r ** 0.5, torch.randn(k_c, n_c, generator=g) / k_c ** 0.5
    out = torch.full((B, k_r * k_c + 3), 7.0, device="cuda")
    split = dtype == torch.float32
    ops().gradproj_dense(G.cuda(), A.cuda(), ops().prepare_projection(P_r.cuda(), split), ops().prepare_projection(P_c.cuda(), split),
                         k_r, k_c, 0.5, out[:, :k_r * k_c])
    after()
    ref = 0.5 * torch.einsum("btr,btc->brc", G.double() @ P_r.double().t(), A.double() @ P_c.double().t())
    # every factor of a product is rounded once: to 8 bits (P of a bf16 layer), or to two parts of 8 bits
    assert O.rel_fro(out[:, :k_r * k_c], ref.flatten(1)) < (2 * 2.0 ** -15 if split else 2 * 2.0 ** -8)
    assert (out[:, k_r * k_c:] == 7.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(1, 3, 5, 1, 1), (2, 63, 1920, 57, 57), (4, 36, 307, 9, 9), (2, 1212, 717, 26, 26), (16, 130, 64, 64, 33),
                                  (40, 128, 230, 16, 16), (90, 200, 136, 32, 64)])
def test_gradproj_embedding_unit_counts_and_widths(case, dtype):
    B, T, d, k_o, k_i = case
    g = torch.Generator().manual_seed(18)
    vocab = 211
    ids = torch.randint(0, vocab, (B, T), generator=g)
    G = torch.randn(B, T, d, generator=g).to(dtype)
    P_o, P_i = torch.randn(k_o, d, generator=g) / k_o ** 0.5, torch.randn(k_i, vocab, generator=g)
    split = dtype == torch.float32
    out = ops().gradproj_embedding(ids.cuda(), G.cuda(), ops().prepare_projection(P_o.cuda(), split),
                                   ops().prepare_embedding_projection(P_i.cuda()), k_o, k_i)
    after()
    ref = torch.einsum("bto,bti->boi", G.double() @ P_o.double().t(), P_i.double().t()[ids])
    assert O.rel_fro(out, ref.flatten(1)) < (2 * 2.0 ** -15 if split else 2 * 2.0 ** -8)


@pytest.mark.parametrize("n_t,n_v,T,F", [(32, 8, 64, 768), (5, 2, 9, 701), (48, 12, 3, 4096)])
def test_kernels_that_start_early_see_what_the_kernel_ahead_wrote(n_t, n_v, T, F):
    """A chain of deterministic reductions, again and again in the same buffers with other values: launched
    as usual, each kernel up while the one ahead still writes, and captured, where the order is plain.  The
    same additions in the same order: the same bits."""
    from ghostsuite_b200 import _lib
    A, G = torch.empty(n_t + n_v, T, F, device="cuda"), torch.empty(n_t + n_v, T, F, device="cuda")

    def chain():
        gw, gb = ops().layernorm_persample(A, G, 1e-5)
        M, Mb = ops().small_gram(gw, n_v), ops().small_gram(gb, n_v)
        s = ops().rows_sum(gw, n_t, 1.0, torch.float32)
        return gw, gb, M, Mb, s, ops().matrix_sum([M, Mb])[:(n_v + 1) * n_t]      # the word behind them is the error word

    gen = torch.Generator(device="cuda").manual_seed(3)
    A.normal_(generator=gen)
    G.normal_(generator=gen)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plain = chain()
    for _ in range(50):
        A.normal_(generator=gen)
        G.normal_(generator=gen)
        early = chain()
        graph.replay()
        for x, y in zip(early, plain):
            assert torch.equal(x, y)
        del early, x
    torch.cuda.synchronize()
    _lib.poll_kernel_error()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n1,n2", [(32 * 65535 + 1, 17), (32 * 65535 + 1, 33), (17, 32 * 65535 + 1)])
def test_similarity_of_more_rows_than_a_grid_has_small_blocks(n1, n2, dtype):
    """The block shape that costs least has no grid for these rows: the next one takes them."""
    d = 8
    gen = torch.Generator(device="cuda").manual_seed(1)
    P1 = torch.randn((n1, d), generator=gen, device="cuda").to(dtype)
    P2 = torch.randn((n2, d), generator=gen, device="cuda").to(dtype)
    got = ops().projection_similarity(P1, P2)
    after()
    # eight products of 16-bit parts and eight additions in float32
    assert O.rel_fro(got.cpu(), (P1.double() @ P2.double().t()).cpu()) < 3e-5


@pytest.mark.parametrize("f32", ["G", "A"])
@pytest.mark.parametrize("case", [(2, 1, 7, 5, 1, 1), (4, 130, 72, 200, 32, 32), (2, 129, 333, 1001, 16, 17), (1, 300, 512, 2944, 44, 44),
                                  (3, 40, 130, 71, 70, 9)])
def test_gradproj_dense_of_mixed_operands(case, f32):
    """One operand float32, the other bf16, on vector boundaries and off them, shared units and whole ones, ranks beyond the
    loaders': the bf16 operand counts as the values it holds, and no copy of it in float32 is made."""
    B, T, n_i, n_o, k_i, k_o = case
    A, G = make(B, T, n_i, n_o, torch.float32, seed=29)
    G, A = (G, A.bfloat16()) if f32 == "G" else (G.bfloat16(), A)
    g = torch.Generator().manual_seed(30)
    P_i, P_o = torch.randn(k_i, n_i, generator=g) / k_i ** 0.5, torch.randn(k_o, n_o, generator=g) / k_o ** 0.5
    o = ops()
    Pr, Pc = o.prepare_projection(P_o.cuda(), True), o.prepare_projection(P_i.cuda(), True)
    out, Gd, Ad = torch.empty((B, k_o * k_i), device="cuda"), G.cuda(), A.cuda()
    o.gradproj_dense(Gd, Ad, Pr, Pc, k_o, k_i, 1.0, out)
    after()
    ref = O.gradproj_dense(A.double(), G.double(), P_i, P_o, compute_dtype=torch.float64) / B
    assert O.rel_fro(out.reshape(B, k_o, k_i), ref) < 1e-4
    made = torch.cuda.memory_stats()["allocation.all.allocated"]
    o.gradproj_dense(Gd, Ad, Pr, Pc, k_o, k_i, 1.0, out)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == made      # workspaces are kept from the first call


@pytest.mark.parametrize("B,T", [(0, 5), (3, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradproj_dense_refuses_an_empty_call(B, T, dtype):
    P = [ops().prepare_projection(torch.ones(4, n, device="cuda"), dtype == torch.float32) for n in (65, 40)]
    with pytest.raises(ValueError):
        ops().gradproj_dense(torch.zeros(B, T, 65, dtype=dtype, device="cuda"), torch.zeros(B, T, 40, dtype=dtype, device="cuda"), P[0], P[1], 4, 4, 1.0)


# Rows that begin anywhere, between values that nothing may take in: every distance of the first row from a 16-byte boundary, pitches of
# all residues, tokens around the eights that loader warps share and the tile, columns around a slice of 128 bytes and a stage of 64;
# stages of both groups of warps, and fewer than groups
@pytest.mark.parametrize("kinds", [("bf16", "bf16"), ("f32", "f32"), ("f32", "bf16"), ("bf16", "f32")])
@pytest.mark.parametrize("case", [(1, 1, 1, 3, 9, 5), (2, 7, 31, 33, 9, 33), (1, 130, 63, 65, 32, 17), (3, 128, 64, 127, 4, 4), (2, 9, 96, 97, 64, 40),
                                  (160, 16, 66, 161, 8, 8), (150, 255, 35, 129, 40, 64), (1, 15, 1021, 700, 33, 64), (20, 33, 515, 258, 12, 12)])
def test_gradproj_rows_that_begin_anywhere(case, kinds):
    B, T, n_r, n_c, k_r, k_c = case
    types = {"bf16": torch.bfloat16, "f32": torch.float32}
    g = torch.Generator(device="cuda").manual_seed(31)
    P_r, P_c = (torch.randn(k, n, generator=g, device="cuda") / k ** 0.5 for k, n in ((k_r, n_r), (k_c, n_c)))
    split = "f32" in kinds
    P = [ops().prepare_projection(x, split) for x in (P_r, P_c)]
    bound = 2 * 2.0 ** -15 if split else 2 * 2.0 ** -8         # as in the test of unit counts and widths
    for offset in range(8):
        x = []
        for kind, n in zip(kinds, (n_r, n_c)):
            buf = torch.full((B * T * n + 16,), float("nan"), device="cuda").to(types[kind])
            view = buf[offset:offset + B * T * n].view(B, T, n)
            view.copy_(torch.randn(B, T, n, generator=g, device="cuda"))
            x.append(view)
        out = ops().gradproj_dense(x[0], x[1], P[0], P[1], k_r, k_c, 1.0, torch.full((B, k_r * k_c), 7.0, device="cuda"))
        after()
        ref = torch.einsum("btr,btc->brc", x[0].double() @ P_r.double().t(), x[1].double() @ P_c.double().t())
        assert O.rel_fro(out.cpu(), ref.flatten(1).cpu()) < bound
        if kinds[0] == kinds[1]:
            ids = torch.randint(0, 50, (B, T), generator=g, device="cuda")
            rows = torch.randn(k_c, 50, generator=g, device="cuda")
            out = ops().gradproj_embedding(ids, x[0], P[0], ops().prepare_embedding_projection(rows), k_r, k_c)
            after()
            ref = torch.einsum("btr,btc->brc", x[0].double() @ P_r.double().t(), rows.double().t()[ids])
            assert O.rel_fro(out.reshape(B, -1).cpu(), ref.flatten(1).cpu()) < bound


# both sides of what sends rows through the ring (16 MB of float32, 128 of bf16, more than 16 rows on either side); one CTA to a block
# of scores; eight splits and nine
@pytest.mark.parametrize("n1,n2,D,dtype", [
    (16, 17, 131072, torch.float32), (17, 17, 131072, torch.float32), (17, 17, 131073, torch.float32), (1100, 1090, 2048, torch.float32),
    (64, 66, 491520 + 8, torch.bfloat16), (64, 66, 500000 + 8, torch.bfloat16), (5, 7, 8 * 1024, torch.float32), (5, 7, 9 * 1024, torch.bfloat16)])
def test_projection_similarity_routes(n1, n2, D, dtype):
    """Also into rows of a wider matrix: nothing beside the scores is written."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(25)
    a, b = (torch.randn(n, D, generator=g, device="cuda").to(dtype) for n in (n1, n2))
    ref = a.double() @ b.double().t()
    bound = 2.0 ** -15 * a.double().norm(dim=1)[:, None] * b.double().norm(dim=1)[None]
    for pitch in (n2, (n2 + 7) // 4 * 4):
        S = torch.full((n1, pitch), 7.0, device="cuda")
        _lib.check(lib.ghost_projection_similarity(a.data_ptr(), b.data_ptr(), 1 if dtype == torch.float32 else 0, n1, n2, D, D, D,
                                                   1.0, S.data_ptr(), pitch, stream))
        after()
        assert ((S[:, :n2].double() - ref).abs() <= bound).all()
        assert (S[:, n2:] == 7.0).all()


# one to three words past the last sixteen bytes and none, results off sixteen bytes, both sides of 16 MB of operands
@pytest.mark.parametrize("offset", [0, 1, 4])
@pytest.mark.parametrize("n1,n2,D", [(3, 7, 250000), (5, 18, 90001), (9, 11, 100008), (16, 32, 20000), (31, 45, 300008),
                                     (5, 18, 173913), (5, 18, 173914), (31, 45, 52628), (31, 45, 52632), (9, 11, 200008)])
def test_projection_similarity_over_old_values(n1, n2, D, offset):
    """Scores that several blocks add up: what was there does not count, and nothing beside them is written."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(31)
    a, b = (torch.randn(n, D, generator=g, device="cuda") for n in (n1, n2))
    buf = torch.full((n1 * n2 + 16,), float("nan"), device="cuda")
    S = buf[offset:offset + n1 * n2]
    for _ in range(2):
        _lib.check(lib.ghost_projection_similarity(a.data_ptr(), b.data_ptr(), 1, n1, n2, D, D, D, 1.0, S.data_ptr(), n2, stream))
    after()
    bound = 2.0 ** -15 * a.double().norm(dim=1)[:, None] * b.double().norm(dim=1)[None]
    assert ((S.view(n1, n2).double() - a.double() @ b.double().t()).abs() <= bound).all()
    assert int(buf.isnan().sum()) == 16


# 8, 19, 24 and 40 MB of split sums: blocks that clear 1024 vectors each, more than the largest grid does in one round (two of
# them), and a memset above 32 MB.  The sums are merged by a launch of their own, so it shows that there are several
@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("rows,m,n", [(6000, 1024, 2048), (16384, 2048, 2432), (16384, 2048, 3072), (32768, 2560, 4096)])
def test_wgrad_split_sums_over_old_values(rows, m, n, mode):
    """Whole numbers whose sums float32 holds: equal whatever the splits, unless old sums count."""
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(32)
    X, Y = (torch.randint(-2, 3, (1, rows, c), generator=g, device="cuda").bfloat16() for c in (m, n))
    ref = X[0].float().t() @ Y[0].float()
    try:
        _lib.check(lib.ghost_set_wgrad_pair_mode(mode))
        for scale in (1.0, 0.25):            # the second one over the sums of the first
            before = _lib.launch_count()
            out = ops().wgrad(X, Y, scale, torch.float32)
            assert _lib.launch_count() - before == (3 if m * n * 4 <= 32 << 20 else 2)
            after()
            assert torch.equal(out, scale * ref)
    finally:
        _lib.check(lib.ghost_set_wgrad_pair_mode(1))


# layers of few rows whose pairs of samples are shared by clusters (long rows): one tile a pair and several, rows that end inside a
# warp's columns, unaligned rows, blocks behind the column sums that fill up a cluster, no gradient
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n_t,n_v,T,d,p", [(4, 12, 1, 109, 9001), (9, 3, 1, 8192, 260), (2, 2, 8, 4096, 33), (3, 2, 16, 5001, 16), (5, 1, 5, 100, 7000)])
def test_few_rows_shared_by_clusters(n_t, n_v, T, d, p, dtype):
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    A, G = (x.cuda() for x in make(n_t + n_v, T, d, p, dtype, seed=35))
    f32 = int(dtype == torch.float32)
    assert lib.ghost_dense_small_fits(f32, n_t, n_v, T, d, p)
    a, g = A.double(), G.double()
    grams = [torch.einsum("vsd,btd->vbst", x[n_t:], x[:n_t]) for x in (a, g, a.abs(), g.abs())]
    # chains of 4 K / 1024 products in each lane, then 31 values of other lanes, warps and blocks; T^2 entries added up
    eps = ((4 * (d // 1024 + p // 1024 + 2)) + 2 * 31 + T * T) * 2.0 ** -24
    bound = eps * (grams[2] * grams[3]).sum((2, 3))
    for want_grad in (True, False):
        assert lib.ghost_dense_small_cluster_size(n_t, n_v, T, d, p, int(want_grad)) > 1
        M = torch.full((n_v, n_t), 7.0, device="cuda")
        grad, sums = torch.full((p, d), 7.0, dtype=dtype, device="cuda"), torch.full((n_t + n_v, p), 7.0, device="cuda")
        _lib.check(lib.ghost_dense_small(A.data_ptr(), G.data_ptr(), f32, n_t, n_v, T, d, p, 0, M.data_ptr(), grad.data_ptr() if want_grad else None,
                                         f32, 0.5, sums.data_ptr() if want_grad else None, torch.cuda.current_stream().cuda_stream))
        after()
        assert ((M.double() - (grams[0] * grams[1]).sum((2, 3))).abs() <= bound).all()
        if want_grad:
            assert O.rel_fro(grad, 0.5 * torch.einsum("ntp,ntd->pd", g[:n_t], a[:n_t])) < (2.0 ** -8 if not f32 else 1e-6)
            assert O.rel_fro(sums, g.sum(1)) < 1e-6


# results that the GEMM writes itself (few rows) and adds up in a workspace: blocks of 32 rows and 32 or 64 columns that end early,
# rows that begin on 16 bytes and anywhere, an unaligned result, old values kept; whole numbers, so exact in every type
@pytest.mark.parametrize("parts,out_dtype", [(1, torch.bfloat16), (1, torch.float32), (2, torch.float32), (2, torch.bfloat16)])
@pytest.mark.parametrize("m,n", [(1, 1), (33, 65), (129, 257), (160, 328), (300, 63), (48, 318), (49, 545)])
@pytest.mark.parametrize("rows", [40, 3000])
def test_train_gradient_stores(rows, m, n, parts, out_dtype):
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    gen = torch.Generator().manual_seed(7)
    X, Y = (torch.zeros(parts, rows, -(-c // 64) * 64, dtype=torch.bfloat16) for c in (m, n))
    X[0, :, :m], Y[0, :, :n] = (torch.randint(-1, 2, (rows, c), generator=gen).bfloat16() for c in (m, n))
    X, Y = X.cuda(), Y.cuda()
    want = X[0, :, :m].double().t() @ Y[0, :, :n].double()
    assert want.abs().max() < 254
    ws = torch.empty(lib.ghost_wgrad_workspace_bytes(m, n), dtype=torch.uint8, device="cuda")
    for first in (0, 1):                              # elements in front of the result
        buf = torch.full((first + m * n + 64,), 2.0, dtype=out_dtype, device="cuda")
        out = buf[first:first + m * n]
        for accumulate in (0, 1):
            _lib.check(lib.ghost_wgrad_parts(X.data_ptr(), Y.data_ptr(), parts, rows, rows, m, n, X.shape[2], Y.shape[2], 1.0 if not accumulate else -1.0,
                                             accumulate, out.data_ptr(), int(out_dtype == torch.float32), ws.data_ptr(), ws.numel(),
                                             torch.cuda.current_stream().cuda_stream))
            after()
            assert torch.equal(out.double().view(m, n), want if not accumulate else 0 * want)
        assert (buf[:first] == 2).all() and (buf[first + m * n:] == 2).all()


# just below 32 MB, 32 MB, more (a memset); a word, two and three behind the last sixteen bytes; results off sixteen bytes
@pytest.mark.parametrize("n_t,n_v,offset", [(4095, 2048, 0), (4096, 2048, 0), (4097, 2048, 0), (4096, 2048, 4), (4096, 2048, 1),
                                            (3, 1, 0), (2, 1, 0), (1, 1, 0), (5, 1, 0), (13, 315, 0), (1024, 4, 0), (1025, 4, 0)])
def test_gram_matrix_over_old_values(n_t, n_v, offset):
    """All of the matrix that the Grams add to is cleared, and nothing beside it is written."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n_t)
    a, b, u, v = (torch.randint(-2, 3, (n, 8), generator=g, device="cuda").bfloat16() for n in (n_t, n_v, n_t, n_v))
    buf = torch.full((n_v * n_t + 16,), float("nan"), device="cuda")
    M = buf[offset:offset + n_v * n_t]
    _lib.check(lib.ghost_gram_dot_bf16(a.data_ptr(), b.data_ptr(), u.data_ptr(), v.data_ptr(), n_t, n_v, 1, 8, 8, 8, 8, 8, 8, 0, 1.0,
                                       M.data_ptr(), stream))
    after()
    assert torch.equal(M.view(n_v, n_t), (b.float() @ a.float().t()) * (v.float() @ u.float().t()))      # whole numbers
    assert int(buf.isnan().sum()) == 16


# one block of tokens and several; a gradient in one split and in several (5000 and 9000 rows), by one CTA or a pair; a matrix of more
# entries than the GEMM's grid has threads (150 x 300 and 400 x 400)
@pytest.mark.parametrize("parts", [1, 2])
@pytest.mark.parametrize("n_t,n_v,T,d,p", [(3, 2, 5, 64, 128), (5, 1, 130, 192, 64), (4, 2, 1250, 256, 128), (9, 1, 1000, 128, 256),
                                           (300, 150, 2, 64, 64), (400, 400, 1, 128, 256)])
def test_gram_pass_entry_point(n_t, n_v, T, d, p, parts):
    """ghost_gram_pass over matrices of old values: Grams with the gradient, whose GEMM clears them, and without; either order of
    the gradient, each kernel; nothing beside the results is written."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n_t)
    N = n_t + n_v
    # whole numbers: exact in any order, and in one bf16 part; the second part (a residual) is then zero
    A, G = (torch.randint(-1, 2, (N * T, c), generator=g, device="cuda").bfloat16() for c in (d, p))
    At, Av, Gt, Gv = A[:n_t * T].float(), A[n_t * T:].float(), G[:n_t * T].float(), G[n_t * T:].float()
    ref = ((Av @ At.t()) * (Gv @ Gt.t())).view(n_v, T, n_t, T).double().sum((1, 3))
    assert ref.abs().max() < 2 ** 24
    if parts == 2:
        A, G = (torch.cat([x, torch.zeros_like(x)]) for x in (A, G))
    size = int(lib.ghost_wgrad_workspace_bytes(max(d, p), max(d, p)))
    ws = torch.full((size,), 0xff, dtype=torch.uint8, device="cuda")
    try:
        for mode in (0, 2):
            _lib.check(lib.ghost_set_wgrad_pair_mode(mode))
            for in_by_out in (0, 1):
                for with_grad, dtype in ((True, torch.float32), (True, torch.bfloat16), (False, torch.float32)):
                    buf = torch.full((n_v * n_t + 16,), float("nan"), device="cuda")
                    M = buf[8:8 + n_v * n_t]
                    shape = (d, p) if in_by_out else (p, d)
                    grad = torch.full(shape, float("nan"), device="cuda", dtype=dtype)
                    _lib.check(lib.ghost_gram_pass(A.data_ptr(), G.data_ptr(), parts, n_t, n_v, T, d, p, d, p, in_by_out, M.data_ptr(), 0.5,
                                                   grad.data_ptr() if with_grad else None, int(dtype == torch.float32), ws.data_ptr(), size, stream))
                    after()
                    assert torch.equal(M.view(n_v, n_t).double(), ref)
                    assert int(buf.isnan().sum()) == 16
                    want = 0.5 * (At.t() @ Gt if in_by_out else Gt.t() @ At)
                    if with_grad:
                        assert torch.equal(grad, want.to(dtype))
                    else:
                        assert bool(grad.isnan().all())
    finally:
        _lib.check(lib.ghost_set_wgrad_pair_mode(1))
    bad = (None, G.data_ptr(), parts, n_t, n_v, T, d, p, d, p, 0, M.data_ptr(), 0.5, None, 1, ws.data_ptr(), size, stream)
    for at, value in ((0, None), (2, 3), (3, 0), (4, 0), (5, 0), (6, 0), (8, d - 8), (11, None)):
        args = list(bad)
        args[0] = A.data_ptr()
        args[at] = value
        assert lib.ghost_gram_pass(*args) != 0


# rows of which 32, 16, 8, four and more than a whole draw's bytes are drawn at once; tables of a part of a draw, one and many
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [8, 384, 392, 1544, 6152])
@pytest.mark.parametrize("vocab", [3, 33, 1025])
def test_embedding_rows_without_tokens_are_zero(vocab, d, dtype):
    """Beside rows that have some: their gradient is the tokens' sum, all others are zero whatever the buffer held."""
    n_t, n_v, T = 3, 1, 5
    g = torch.Generator(device="cuda").manual_seed(8)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=g, device="cuda")
    G = torch.randn((n_t + n_v, T, d), generator=g, device="cuda").to(dtype)
    ref = torch.zeros((vocab, d), dtype=torch.float64, device="cuda")
    ref.index_add_(0, ids[:n_t].flatten(), G[:n_t].flatten(0, 1).double())
    for _ in range(2):
        held = torch.full((vocab, d), float("nan"), device="cuda", dtype=dtype)      # the buffer that the result may get
        del held
        grad = ops().embedding_wgrad(ids[:n_t], G[:n_t], n_t, vocab, 1.0, 1.0)
        after()
        # up to 15 tokens a row: the sum is float32, rounded once
        assert ((grad.double() - ref).abs() <= (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -20) * (1 + ref.abs())).all()
        empty = torch.ones(vocab, dtype=torch.bool, device="cuda")
        empty[ids[:n_t].flatten()] = False
        assert (grad[empty] == 0).all()


def _rows(samples, T, cols, ld, seed):
    """bf16 rows of `cols` columns in rows of `ld`, NaN between them: whoever reads past a row shows it."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.full((samples, T, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
    x[..., :cols] = torch.randn((samples, T, cols), generator=g, device="cuda").bfloat16()
    return x


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n_t,n_v,T,ka,kg", [(3, 2, 5, 24, 17), (5, 1, 130, 64, 40), (3, 2, 257, 200, 136)])
def test_gram_entry_point_on_four_buffers(n_t, n_v, T, ka, kg, mode):
    """ghost_gram_dot_bf16 as a C caller has it: train and validation rows in buffers of their own, every one with
    its own pitch, either rounding, each kernel."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    up = lambda n: (n + 7) // 8 * 8
    ld = (up(ka), up(ka) + 8, up(kg) + 16, up(kg))
    at, av = _rows(n_t, T, ka, ld[0], 1), _rows(n_v, T, ka, ld[1], 2)
    gt, gv = _rows(n_t, T, kg, ld[2], 3), _rows(n_v, T, kg, ld[3], 4)
    a = torch.einsum("btk,vsk->vbst", at[..., :ka].double(), av[..., :ka].double())
    g = torch.einsum("btk,vsk->vbst", gt[..., :kg].double(), gv[..., :kg].double())
    try:
        _lib.check(lib.ghost_set_gram_pair_mode(mode))
        for rounding in (0, 1):
            M = torch.full((n_v, n_t), float("nan"), device="cuda")
            _lib.check(lib.ghost_gram_dot_bf16(at.data_ptr(), av.data_ptr(), gt.data_ptr(), gv.data_ptr(), n_t, n_v, T, ka, kg,
                                               *ld, rounding, 0.5, M.data_ptr(), stream))
            after()
            # products of bf16 values are exact, sums float32; rounded entries carry three roundings of 2^-9
            assert O.rel_fro(M, 0.5 * (a * g).sum((2, 3))) < (1e-4 if rounding == 0 else 2e-2)
    finally:
        _lib.check(lib.ghost_set_gram_pair_mode(1))


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("rows,m,n", [(7, 24, 17), (300, 256, 320), (5000, 72, 130), (9000, 256, 64)])
def test_wgrad_entry_point_on_strided_rows(rows, m, n, mode):
    """ghost_wgrad_bf16 on rows inside wider ones, written and accumulated, in either type, in one split and several."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    ldx, ldy = (m + 7) // 8 * 8 + 8, (n + 7) // 8 * 8 + 24
    X, Y = _rows(1, rows, m, ldx, 5), _rows(1, rows, n, ldy, 6)
    ref = 0.25 * X[0, :, :m].double().t() @ Y[0, :, :n].double()
    size = int(lib.ghost_wgrad_workspace_bytes(m, n))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    try:
        _lib.check(lib.ghost_set_wgrad_pair_mode(mode))
        for dtype in (torch.float32, torch.bfloat16):
            for accumulate in (0, 1):
                out = torch.full((m, n), 2.0 if accumulate else float("nan"), device="cuda", dtype=dtype)
                _lib.check(lib.ghost_wgrad_bf16(X.data_ptr(), Y.data_ptr(), rows, m, n, ldx, ldy, 0.25, accumulate, out.data_ptr(),
                                                1 if dtype == torch.float32 else 0, ws.data_ptr(), size, stream))
                after()
                assert O.rel_fro(out, ref + 2.0 * accumulate) < (1e-4 if dtype == torch.float32 else 1e-2)
    finally:
        _lib.check(lib.ghost_set_wgrad_pair_mode(1))


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("n_t,n_v,T,m,n", [(3, 2, 5, 24, 17), (5, 9, 70, 256, 320), (33, 1, 9, 72, 130)])
def test_persample_entry_point_on_strided_rows(n_t, n_v, T, m, n, mode):
    """ghost_persample_dot_bf16 on rows inside wider ones: bf16 tiles with the column sums of either operand, and
    float32 tiles of the three stacked parts that ghost_cast_split_bf16 makes of float32 rows."""
    from ghostsuite_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    N = n_t + n_v
    ldx, ldy = (m + 7) // 8 * 8 + 8, (n + 7) // 8 * 8 + 16

    def call(X, Y, tokens, ldx, ldy, f32, colsum_of, sums):
        size = int(lib.ghost_persample_workspace_bytes(n_t, n_v, m, n, f32))
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        M, grad = torch.full((n_v, n_t), float("nan"), device="cuda"), torch.full((m, n), float("nan"), device="cuda")
        _lib.check(lib.ghost_persample_dot_bf16(X.data_ptr(), Y.data_ptr(), n_t, n_v, tokens, m, n, ldx, ldy, 2.0, M.data_ptr(), f32,
                                                grad.data_ptr(), 1, 0.5, 0, colsum_of, sums.data_ptr() if colsum_of else None,
                                                ws.data_ptr(), size, stream))
        after()
        return M, grad

    def reference(x, y):
        w = torch.einsum("btm,btn->bmn", x.double(), y.double())
        return 2.0 * torch.einsum("vmn,bmn->vb", w[n_t:], w[:n_t]), 0.5 * w[:n_t].sum(0)

    try:
        _lib.check(lib.ghost_set_persample_pair_mode(mode))
        X, Y = _rows(N, T, m, ldx, 7), _rows(N, T, n, ldy, 8)
        M_ref, grad_ref = reference(X[..., :m], Y[..., :n])
        for colsum_of in (0, 1, 2):
            sums = torch.full((N, n if colsum_of == 2 else m), float("nan"), device="cuda")
            M, grad = call(X, Y, T, ldx, ldy, 0, colsum_of, sums)
            assert O.rel_fro(M, M_ref) < 2e-2 and O.rel_fro(grad, grad_ref) < 2e-2     # tiles in bf16
            if colsum_of:
                assert O.rel_fro(sums, (X[..., :m] if colsum_of == 1 else Y[..., :n]).double().sum(1)) < 1e-5
        g = torch.Generator(device="cuda").manual_seed(9)
        x, y = torch.randn((N, T, m), generator=g, device="cuda"), torch.randn((N, T, n), generator=g, device="cuda")
        stacked = []
        for src, ld, kinds in ((x, ldx, (0, 1, 0)), (y, ldy, (0, 0, 1))):
            cols = src.shape[-1]
            dst = torch.full((N, 3 * T, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
            _lib.check(lib.ghost_cast_split_bf16(src.data_ptr(), 1, N, T, cols, cols, dst.data_ptr(), ld, (cols + 7) // 8 * 8, 3, *kinds, 1, stream))
            stacked.append(dst)
        M_ref, grad_ref = reference(x, y)
        M, grad = call(*stacked, 3 * T, ldx, ldy, 1, 0, None)
        assert O.rel_fro(M, M_ref) < 1e-4 and O.rel_fro(grad, grad_ref) < 1e-4
    finally:
        _lib.check(lib.ghost_set_persample_pair_mode(1))

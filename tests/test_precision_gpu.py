"""Accuracy of the sums against 64 bits, at lengths where the order of a sum shows.

The tensor core adds into an accumulator that it truncates, so a long chain of products of one sign
comes out too small by up to 2^-23 per product added (2^-24 on average); float32 additions round to
nearest and leave no such bias.  The data are therefore positive and the tests look at the mean signed
error over many entries: chains of a few products stay below 2^-23, rounding averages out."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BIAS = 2.0 ** -23


def ops():
    from ghostsuite_b200 import ops as _ops
    return _ops


def positive(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (0.5 + torch.rand(shape, generator=g, device="cuda")).to(dtype)


def bias(got, want):
    want = want.double()
    return ((got.double() - want) / want).mean().abs().item()


# text-like ids (every validation token of an id in one list) and one id above the summed-rows line; feature
# counts on both sides of one load step
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [256, 731, 2048])
@pytest.mark.parametrize("vocab", [1, 40])
def test_embedding_matrix(vocab, d, dtype):
    n_t, n_v, T = 16, 8, 48
    g = torch.Generator(device="cuda").manual_seed(3)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=g, device="cuda")
    G = positive((n_t + n_v, T, d), dtype, 4)
    M = ops().embedding_dot(ids, G, n_v, vocab)
    R = torch.zeros(n_t + n_v, vocab, d, dtype=torch.float64, device="cuda")
    for i in range(n_t + n_v):
        R[i].index_add_(0, ids[i], G[i].double())
    R = R.reshape(n_t + n_v, -1)
    assert bias(M, R[n_t:] @ R[:n_t].t()) < BIAS


def test_embedding_matrix_beyond_one_block():
    """More entries than a block sums in shared memory; groups of train samples through the C entry."""
    n_t, n_v, T, d, vocab = 300, 20, 6, 64, 9
    g = torch.Generator(device="cuda").manual_seed(5)
    ids = torch.randint(0, vocab, (n_t + n_v, T), generator=g, device="cuda")
    ids[:, 0] = 4                        # every pair shares an id: the errors below are relative to the entry
    G = positive((n_t + n_v, T, d), torch.float32, 6)
    R = torch.zeros(n_t + n_v, vocab, d, dtype=torch.float64, device="cuda")
    for i in range(n_t + n_v):
        R[i].index_add_(0, ids[i], G[i].double())
    R = R.reshape(n_t + n_v, -1)
    want = 0.5 * R[n_t:] @ R[:n_t].t()
    M = ops().embedding_dot(ids, G, n_v, vocab, 0.5)
    # a dot product of 64 terms in float32, then 64-bit sums: 2^-24 per addition of the longest chain
    assert ((M.double() - want) / want).abs().max() < 8 * BIAS and bias(M, want) < BIAS
    from ghostsuite_b200 import _lib
    lib = _lib.load()
    room = int(lib.ghost_embedding_dot_workspace_bytes_for(n_v, T, vocab, d))       # groups of 32
    ws = torch.empty(room, dtype=torch.uint8, device="cuda")
    M2 = torch.full_like(M, 7.0)
    _lib.check(lib.ghost_embedding_dot(ids.data_ptr(), G.data_ptr(), 1, n_t, n_v, T, d, vocab, 0.5, M2.data_ptr(),
                                       ws.data_ptr(), room, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert ((M2.double() - want) / want).abs().max() < 8 * BIAS


# float32 results: no chain longer than what the split of the rows allows (products of 16 rows each)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,n,chain", [(64, 64, 4), (256, 256, 8), (768, 768, 32), (1000, 768, 64)])
def test_wgrad_float32_result(m, n, chain, dtype):
    rows = 4096
    X, Y = positive((rows, m), dtype, 1), positive((rows, n), dtype, 2)
    W = ops().wgrad(X, Y, 1.0, torch.float32)
    parts = 3 if dtype == torch.float32 else 1              # hi.hi, lo.hi and hi.lo go to one accumulator
    assert bias(W, X.double().t() @ Y.double()) < parts * chain / 2 * BIAS


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dim", [9999, 98304])
@pytest.mark.parametrize("n1,n2", [(8, 8), (16, 64), (32, 32), (64, 64), (100, 7), (128, 20), (3, 100)])
def test_similarity(n1, n2, dim, dtype):
    a, b = positive((n1, dim), dtype, 1), positive((n2, dim), dtype, 2)
    S = ops().projection_similarity(a, b)
    assert bias(S, a.double() @ b.double().t()) < BIAS


@pytest.mark.parametrize("F", [768, 50257])
def test_end_of_pass_gram(F):
    """Root mean square error of the matrix of per-sample vectors.  256 accumulators a pair take F / 256
    products each and are added in pairs.  An addition rounds by 0.29 units in the last place on average,
    2^-23 / m of a sum whose mantissa is m (the same at every level of the pairs); the squares of the levels
    add up to twice the last one's.  A quarter on top for the spread of the mantissas."""
    X = positive((256 + 32, F), torch.float32, 7)
    M = torch.empty(32, 256, device="cuda")
    ops().pass_reduce([{"X": X, "n_train": 256, "n_val": 32, "M": M}], [])
    want = X[256:].double() @ X[:256].double().t()
    rms = ((M.double() - want) / want).pow(2).mean().sqrt().item()
    m = want.mean().item()
    one = 0.29 * BIAS / (m / 2.0 ** math.floor(math.log2(m)))
    assert rms < 1.25 * one * (2 + F / 256 / 3 / 256) ** 0.5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("N,T,F,splits", [(148, 1024, 1032, 2), (148, 1024, 731, 2), (148, 512, 4104, 1), (40, 160, 2048, 7)])
def test_wide_norm_vectors(N, T, F, splits, rms, dtype):
    """Sums over the tokens of terms of either sign: the partial sums grow with the root of their length, so n additions
    in a row leave 2.45e-8 (0.29 ulp of a sum with an average mantissa) times the root of n / 2 of the
    result.  32 rows in registers, the groups of a split, the splits; each term carries another eight
    roundings (mean, variance, root, products).  Half on top."""
    g = torch.Generator(device="cuda").manual_seed(9)
    A, G = (torch.randn((N, T, F), generator=g, device="cuda").to(dtype) for _ in range(2))
    got, _ = ops().layernorm_persample(A, G, 1e-5, rms=rms)
    num = den = 0.0
    for n in range(N):
        x = A[n].double()
        if not rms:
            x = x - x.mean(-1, keepdim=True)
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)
        want = (G[n].double() * x).sum(0)
        num += (got[n].double() - want).pow(2).sum().item()
        den += want.pow(2).sum().item()
    rows = T / splits
    bound = 2.45e-8 * (min(rows, 32) / 2 + rows / 32 / 2 + splits / 2 + 8) ** 0.5
    assert (num / den) ** 0.5 < 1.5 * bound

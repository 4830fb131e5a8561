"""The one-launch CG (FP64 and the FP32 inner CG) at the edges of its row and
shared-memory splits, against plain CG in numpy.

A few iterations on a diagonally dominant matrix (condition number below 4):
every iterate of two correctly coded CGs agrees to a few hundred rounding
errors, so 1e-12 of the largest entry is a wide bound for FP64.  The mixed
solver is held to its own stop: the true FP64 residual.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from arcanefem_gb300 import fem

pytestmark = pytest.mark.gpu

SMS = 152
FULL = SMS * 512          # rows of one row a thread


def matrix(n, longest=7, seed=0):
    """Symmetric, diagonally dominant; with `longest` > 7 one row in 96 has that many entries."""
    rng = np.random.default_rng(seed)
    m = 3 * n
    i = rng.integers(0, n, m)
    j = (i + rng.integers(1, max(2, min(n, 5000)), m)) % n
    if longest > 7:
        heads = np.arange(0, n, 96)
        i = np.concatenate([i, np.repeat(heads, longest - 7)])
        j = np.concatenate([j, (np.repeat(heads, longest - 7) + np.tile(np.arange(1, longest - 6), heads.size)) % n])
    off = i != j
    v = -rng.uniform(0.5, 1.0, off.sum())
    A = sp.coo_matrix((v, (i[off], j[off])), shape=(n, n)).tocsr()
    A = (A + A.T).tocsr()
    d = 2.0 * np.asarray(abs(A).sum(1)).ravel() + 1.0
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A


def block_matrix(nb, seed=0):
    """The same pattern with 3x3 blocks."""
    B = matrix(nb, seed=seed)
    rng = np.random.default_rng(seed + 1)
    K = sp.kron(B, np.ones((3, 3)), format="csr")
    K.data *= rng.uniform(0.9, 1.0, K.nnz)
    K = (K + K.T).tocsr()
    K = (K + sp.diags(2.0 * np.asarray(abs(K).sum(1)).ravel())).tocsr()
    K.sort_indices()
    return K


def cg(A, b, iters):
    x = np.zeros_like(b)
    dinv = 1.0 / A.diagonal()
    r = b.copy()
    z = dinv * r
    p, rz = z.copy(), r @ z
    for _ in range(iters):
        q = A @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = dinv * r
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x


def dev(A):
    return (torch.as_tensor(A.indptr.astype(np.int32), device="cuda"),
            torch.as_tensor(A.indices.astype(np.int32), device="cuda"), torch.as_tensor(A.data, device="cuda"))


@pytest.mark.parametrize("n,longest", [(1, 7), (2, 7), (31, 7), (33, 7), (129, 7), (257, 7), (3072, 7), (3073, 7),
                                       (5000, 7), (FULL, 7),
                                       (FULL + 1, 7), (2 * FULL + 33, 7), (4 * FULL + 1, 7), (6 * FULL, 7),
                                       (6 * FULL + 1, 7), (3000, 300), (20000, 200), (300001, 120)])
def test_iterates_match_numpy(cuda_ctx, n, longest):
    A = matrix(n, min(longest, n), seed=n % 97)
    b = np.random.default_rng(n).standard_normal(n)
    iters = min(6, n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    opt = fem.solver_options(rtol=0.0, atol=1e-300, max_iter=iters)
    try:
        info = fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x, options=opt)
    except fem.AfemError as e:        # max_iter, or an exact zero residual at the smallest sizes
        info = e.info
    want = cg(A, b, info.iterations)
    assert n < 3 or info.iterations == iters
    got = x.cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


# blocks that gather from few others, which the barrier alone waits for: none (a diagonal), the next ones, and a slow
# block with long rows that its neighbours leave behind
@pytest.mark.parametrize("n,width,heavy", [(5000, 0, 0), (FULL + 1, 1, 0), (2 * FULL + 33, 1, 40), (20000, 300, 0),
                                           (20000, 1, 64)])
def test_iterates_of_band_matrices_match_numpy(cuda_ctx, n, width, heavy):
    rng = np.random.default_rng(n + width)
    A = sp.diags([-rng.uniform(0.5, 1.0, n - width)], [width], shape=(n, n)) if width else sp.csr_matrix((n, n))
    if heavy:
        i, j = np.repeat(np.arange(heavy), 1500), np.tile(np.arange(heavy, heavy + 1500), heavy)
        A = A + sp.coo_matrix((-rng.uniform(0.0, 0.01, i.size), (i, j)), shape=(n, n))
    A = (A + A.T).tocsr()
    A = (A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + rng.uniform(1.0, 3.0, n))).tocsr()
    A.sort_indices()
    b = rng.standard_normal(n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    try:
        info = fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                                options=fem.solver_options(rtol=0.0, atol=1e-300, max_iter=10 if width or heavy else 1))
    except fem.AfemError as e:
        info = e.info
    want = cg(A, b, info.iterations)
    assert np.max(np.abs(x.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("n,longest", [(33, 7), (3000, 300), (5000, 7), (FULL + 1, 7), (6 * FULL, 7), (300001, 120)])
def test_mixed_reaches_its_tolerance(cuda_ctx, n, longest):
    A = matrix(n, longest, seed=3)
    b = np.random.default_rng(n).standard_normal(n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                     options=fem.solver_options(rtol=1e-11, max_iter=500, precision=fem.PRECISION_MIXED))
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("nb", [1, 11, 160, 1024, 1025, 1700, FULL // 3 + 1, 60000])
def test_mixed_blocks_reach_their_tolerance(cuda_ctx, nb):
    A = block_matrix(nb)
    n = 3 * nb
    b = np.random.default_rng(n).standard_normal(n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                     options=fem.solver_options(rtol=1e-11, max_iter=500, precision=fem.PRECISION_MIXED, block_size=3))
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-11 * np.linalg.norm(b)


def test_long_solves_span_several_launches(cuda_ctx):
    n = 3000                                    # a chain: about n iterations, more than one launch's
    A = sp.diags([-np.ones(n - 1), 2.0 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    b = np.random.default_rng(0).standard_normal(n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                            options=fem.solver_options(rtol=1e-8, max_iter=200000))
    assert info.iterations > 2000
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-8 * np.linalg.norm(b)


def test_unused_slots_of_a_padded_view(cuda_ctx):
    """Negative columns (unused slots) are zero weights, in and out of shared memory."""
    n = 4000
    A = matrix(n, seed=5)
    width = int(np.diff(A.indptr).max()) + 2
    cols = np.full((n, width), -1, np.int32)
    vals = np.full((n, width), 1e6)
    for i in range(n):
        k = A.indptr[i + 1] - A.indptr[i]
        cols[i, 1:1 + k] = A.indices[A.indptr[i]:A.indptr[i + 1]]
        vals[i, 1:1 + k] = A.data[A.indptr[i]:A.indptr[i + 1]]
    rp = torch.arange(0, n * width + 1, width, dtype=torch.int32, device="cuda")
    b = np.random.default_rng(1).standard_normal(n)
    for precision in (fem.PRECISION_FP64, fem.PRECISION_MIXED):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        fem.cg_solve_csr(cuda_ctx, rp, torch.as_tensor(cols.ravel(), device="cuda"),
                         torch.as_tensor(vals.ravel(), device="cuda"), torch.as_tensor(b, device="cuda"), x,
                         options=fem.solver_options(rtol=1e-11, max_iter=500, precision=precision))
        assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-11 * np.linalg.norm(b)

"""The one-launch CG where it can fail without a wrong number: a block that
never arrives, iterates asked for and not made, and inner solves that take more
than one launch.  Sizes follow the device's SM count."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from arcanefem_gb300 import fem
from test_gpu_cg_resident import block_matrix, cg, dev, matrix

pytestmark = pytest.mark.gpu

BAD_ARG, NOT_CONVERGED, TIMEOUT = 1, 3, 5
OPTIONS = {"fp64": dict(precision=fem.PRECISION_FP64), "mixed": dict(precision=fem.PRECISION_MIXED),
           "blocks": dict(precision=fem.PRECISION_MIXED, block_size=3)}


def rows_of_one_a_thread():
    return min(torch.cuda.get_device_properties(0).multi_processor_count, 256) * 512


# 40 blocks of 128 rows, or 27 of 64 block rows
@pytest.mark.parametrize("form", list(OPTIONS))
@pytest.mark.parametrize("stall", [0, 17, 26])
def test_a_block_that_never_arrives_is_a_timeout(cuda_ctx, form, stall):
    A = block_matrix(1700) if form == "blocks" else matrix(5000)
    n = A.shape[0]
    b = torch.as_tensor(np.random.default_rng(1).standard_normal(n), device="cuda")
    start = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda")
    x, sys = start.clone(), dev(A)
    opt = fem.solver_options(rtol=1e-10, max_iter=500, **OPTIONS[form])
    assert fem.cg_failure_test(cuda_ctx, *sys, b, x, opt, stall, 20000) == TIMEOUT
    assert torch.equal(x, start)
    info = fem.cg_solve_csr(cuda_ctx, *sys, b, x, options=opt)     # the context is still good
    assert info.status == 0 and info.iterations > 0
    assert np.linalg.norm(b.cpu().numpy() - A @ x.cpu().numpy()) <= 1.01e-10 * np.linalg.norm(b.cpu().numpy())


def test_systems_without_polls_have_no_failure_test(cuda_ctx):
    A = matrix(2000)                                # one cluster
    b = torch.ones(2000, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    assert fem.cg_failure_test(cuda_ctx, *dev(A), b, x, fem.solver_options(), 0, 1000) == BAD_ARG
    A = matrix(5000)
    b = torch.ones(5000, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    assert fem.cg_failure_test(cuda_ctx, *dev(A), b, x, fem.solver_options(), 40, 1000) == BAD_ARG


def solve_exactly(ctx, A, b, iters):
    """x after `iters` iterations; anything else that the solve says is an error."""
    x = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    with pytest.raises(fem.AfemError) as e:
        fem.cg_solve_csr(ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                         options=fem.solver_options(rtol=0.0, atol=1e-300, max_iter=iters))
    assert e.value.status == NOT_CONVERGED and e.value.info.iterations == iters
    return x.cpu().numpy()


# the device's edges of one, four and six rows a thread, and the first system past them; iterates as in
# test_gpu_cg_resident.py, to its 1e-12
@pytest.mark.parametrize("rows,more", [(1, 0), (1, 1), (2, 33), (4, 1), (6, 0), (6, 1)])
def test_iterates_at_the_splits_of_this_device(cuda_ctx, rows, more):
    n = rows * rows_of_one_a_thread() + more
    A = matrix(n, seed=n % 97)
    b = np.random.default_rng(n).standard_normal(n)
    want = cg(A, b, 6)
    assert np.max(np.abs(solve_exactly(cuda_ctx, A, b, 6) - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("n,width,heavy", [(5000, 1, 0), (20000, 300, 0), (20000, 1, 64), (170000, 1, 40)])
def test_band_matrices_make_the_iterations_asked_for(cuda_ctx, n, width, heavy):
    rng = np.random.default_rng(n + width)
    A = sp.diags([-rng.uniform(0.5, 1.0, n - width)], [width], shape=(n, n))
    if heavy:
        i, j = np.repeat(np.arange(heavy), 1500), np.tile(np.arange(heavy, heavy + 1500), heavy)
        A = A + sp.coo_matrix((-rng.uniform(0.0, 0.01, i.size), (i, j)), shape=(n, n))
    A = (A + A.T).tocsr()
    A = (A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + rng.uniform(1.0, 3.0, n))).tocsr()
    A.sort_indices()
    b = rng.standard_normal(n)
    want = cg(A, b, 10)
    assert np.max(np.abs(solve_exactly(cuda_ctx, A, b, 10) - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("n", [2000, 5000])
def test_mixed_inner_solves_span_several_launches(cuda_ctx, n):
    """A shifted chain: in numpy the FP32 cycles take 3000 to 4500 iterations at 5000 rows; a launch makes 1890
    there, 1930 at 2000."""
    A = sp.diags([-np.ones(n - 1), (2.0 + 1e-6) * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    b = np.random.default_rng(0).standard_normal(n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                            options=fem.solver_options(rtol=1e-8, max_iter=200000, inner_rtol=1e-3,
                                                       precision=fem.PRECISION_MIXED))
    assert info.status == 0
    if n == 5000:
        assert info.iterations > 2000 * info.refinements
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-8 * np.linalg.norm(b)


def hub_matrix(n, longest, blocks=False):
    """A chain one of whose rows has `longest` entries, as of a node with far more neighbours than the others."""
    rng = np.random.default_rng(longest)
    j = rng.choice(np.arange(2, n - 1), longest, replace=False)
    A = sp.diags([-np.ones(n - 1)], [1], shape=(n, n)) + sp.coo_matrix((np.full(longest, -0.01),
                                                                        (np.zeros(longest, int), j)), shape=(n, n))
    A = (A + A.T).tocsr()
    A = (A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1e-3)).tocsr()
    if blocks:
        A = sp.kron(A, np.array([[2.0, 0.5, 0.25], [0.5, 2.0, 0.5], [0.25, 0.5, 2.0]])).tocsr()
    A.sort_indices()
    return A


# a slice as long as one row: in a cluster and past it, in shared memory and (from about 800 and 900 entries) not
@pytest.mark.parametrize("form", ["mixed", "blocks"])
@pytest.mark.parametrize("n,longest", [(1000, 120), (1000, 950), (9000, 700), (9000, 6000), (90000, 3000)])
def test_mixed_solves_with_one_long_row(cuda_ctx, form, n, longest):
    A = hub_matrix(n, longest, form == "blocks")
    b = np.random.default_rng(n).standard_normal(A.shape[0])
    x = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    info = fem.cg_solve_csr(cuda_ctx, *dev(A), torch.as_tensor(b, device="cuda"), x,
                            options=fem.solver_options(rtol=1e-10, max_iter=20000, **OPTIONS[form]))
    assert info.status == 0 and info.iterations > 0
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01e-10 * np.linalg.norm(b)


def test_a_long_row_costs_fp32_no_more_than_fp64(cuda_ctx):
    """An iteration waits for the longest row.  Walked entry by entry with its values' conversions, one of 15000 took
    the mixed form 1.4 times an FP64 iteration; from the sliced copy 0.8 times."""
    A = hub_matrix(20000, 15000)
    sys, b = dev(A), torch.as_tensor(np.random.default_rng(0).standard_normal(20000), device="cuda")
    best = {}
    for form in ("fp64", "mixed"):
        for _ in range(3):
            x = torch.zeros_like(b)
            info = fem.cg_solve_csr(cuda_ctx, *sys, b, x, options=fem.solver_options(rtol=1e-8, max_iter=20000,
                                                                                    **OPTIONS[form]))
            best[form] = min(best.get(form, np.inf), info.solve_ms / info.iterations)
    assert best["mixed"] <= 1.1 * best["fp64"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("side", [30, 100])
def test_tiny_systems_converge_as_their_multiples(cuda_ctx, side, precision):
    """The same problem at 2^-k: powers of two change no digit in FP64, nor in FP32 until the squares of the residual's
    entries (2^-64 at 2^-44 and 1e-6) leave its normal numbers; they keep 13 bits and more down to 2^-48."""
    T = sp.diags([-np.ones(side - 1), 2.0 * np.ones(side), -np.ones(side - 1)], [-1, 0, 1])
    A = (sp.kron(T, sp.identity(side)) + sp.kron(sp.identity(side), T)).tocsr()
    A.sort_indices()
    sys, b0 = dev(A), np.random.default_rng(0).standard_normal(side * side)
    iters = {}
    for k in (0, 40, 44, 46, 48) + ((200, 400, 460, 480) if precision == "fp64" else ()):
        b = b0 * 2.0 ** -k
        x = torch.zeros(side * side, dtype=torch.float64, device="cuda")
        info = fem.cg_solve_csr(cuda_ctx, *sys, torch.as_tensor(b, device="cuda"), x,
                                options=fem.solver_options(rtol=1e-6, max_iter=1000, **OPTIONS[precision]))
        assert info.status == 0
        iters[k] = info.iterations
        scaled = x.cpu().numpy() * 2.0 ** k
        assert np.linalg.norm(b0 - A @ scaled) <= 1.01e-6 * np.linalg.norm(b0)
    spread = 1.05 if precision == "mixed" else 1.0
    assert max(iters.values()) <= spread * iters[0]

"""The one-launch CG where a block never arrives."""
import numpy as np
import pytest
import torch

from arcanefem_gb300 import fem
from test_gpu_cg_resident import block_matrix, dev, matrix

pytestmark = pytest.mark.gpu

BAD_ARG, TIMEOUT = 1, 5
OPTIONS = {"fp64": dict(precision=fem.PRECISION_FP64), "mixed": dict(precision=fem.PRECISION_MIXED),
           "blocks": dict(precision=fem.PRECISION_MIXED, block_size=3)}


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

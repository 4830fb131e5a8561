"""The reference-rounding element kernels whose products run on the integer
pipe, bit for bit against the oracle where that path has its edges: cells with
exact zeros (unjittered meshes, coordinates on the axes), coordinates near and
beyond the range it takes (scaled by powers of two), cells inside and outside
it in one warp, and cell counts around a warp and a block."""
import numpy as np
import pytest
import torch

from arcanefem_gb300 import fem, meshgen
from oracle import oracle as O
from test_gpu_parity import build_format

pytestmark = pytest.mark.gpu


@pytest.fixture
def own_ctx():
    """A context of the test's own: overflowing cells raise its degenerate-cell flag."""
    ctx = fem.Context()
    yield ctx
    ctx.close()


def assert_bit_exact(got, ref, what):
    """Every entry equal; a cell whose products overflow gives NaN in both."""
    if not np.array_equal(got, ref, equal_nan=True):
        d = ~((got == ref) | (np.isnan(got) & np.isnan(ref)))
        k = int(np.argmax(d))
        raise AssertionError(f"{what}: {int(d.sum())} of {got.size} entries differ; first at {k}: {got[k]!r} vs {ref[k]!r}")


def moved_mesh(make, n, jitter, case):
    m = make(n, jitter=jitter, seed=n)
    x = m.coords.copy()
    if case == "mixed":      # scattered tiny and huge coordinates: their cells leave the integer path's range
        rng = np.random.default_rng(n)
        some = rng.choice(m.nb_node, max(1, m.nb_node // 12), replace=False)
        x[some] *= np.where(np.arange(some.size) % 2 == 0, 2.0 ** -104, 2.0 ** 101)[:, None]
    else:
        x *= 2.0 ** case
    return meshgen.Mesh(m.dim, x, m.cells, m.groups)


CASES = [(1, 0.15, 0), (3, 0.0, 0), (4, 0.15, -70), (4, 0.0, -97), (4, 0.15, -99), (4, 0.15, 99), (5, 0.15, -120),
         (5, 0.15, 110), (6, 0.15, "mixed"), (9, 0.15, 0)]


def oracle_values(m, kind, coeff=None, **kw):
    ptr, nc, _ = O.node_cell(m.nb_node, m.cells)
    rp, cols = O.sparsity(m.nb_node, m.cells)
    with np.errstate(all="ignore"):
        return O.assemble(kind, m.coords, m.cells, ptr, nc, rp, cols, cell_coeff=coeff, **kw)


@pytest.mark.parametrize("n,jitter,case", CASES)
def test_tetrahedra_over_the_operand_ranges(own_ctx, n, jitter, case):
    m = moved_mesh(meshgen.unit_cube_tet, n, jitter, case)
    f = build_format(own_ctx, m)
    f.assemble_poisson()
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_TET4), "tetrahedra")
    k = np.exp(np.random.default_rng(0).standard_normal(m.nb_cell))
    f.assemble_poisson(torch.as_tensor(k, device="cuda"))
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_TET4, coeff=k), "coefficient")


@pytest.mark.parametrize("n,jitter,case", CASES)
def test_hexahedra_over_the_operand_ranges(own_ctx, n, jitter, case):
    m = moved_mesh(meshgen.unit_cube_hex, n, jitter, case)
    f = build_format(own_ctx, m)
    f.assemble_poisson()
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_HEXA8), "hexahedra")
    k = np.exp(np.random.default_rng(0).standard_normal(m.nb_cell))
    f.assemble_poisson(torch.as_tensor(k, device="cuda"))
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_HEXA8, coeff=k), "coefficient")


@pytest.mark.parametrize("lam,mu", [(1.3, 0.7), (0.0, 1.0), (2.0 ** 190, 2.0 ** -190), (2.0 ** 205, 1.0)])
@pytest.mark.parametrize("n,jitter,case", CASES)
def test_elasticity_over_the_operand_ranges(own_ctx, n, jitter, case, lam, mu):
    m = moved_mesh(meshgen.unit_cube_tet, n, jitter, case)
    f = build_format(own_ctx, m, 3)
    f.assemble_elasticity(lam, mu)
    ref = oracle_values(m, O.ELASTICITY_TET4, lam=lam, mu=mu)
    assert_bit_exact(f.values.cpu().numpy(), ref, "elasticity")


@pytest.mark.parametrize("bent", [False, True])
@pytest.mark.parametrize("n,jitter,case", CASES)
def test_triangles_over_the_operand_ranges(own_ctx, n, jitter, case, bent):
    m = moved_mesh(meshgen.unit_square_tri, 3 * n, jitter, case)
    if bent:                     # a third of the nodes out of the plane: their triangles take the general area
        m.coords[::3, 2] = 0.3 * m.coords[::3, 0]
    f = build_format(own_ctx, m)
    f.assemble_poisson()
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_TRI3), "triangles")
    k = np.exp(np.random.default_rng(0).standard_normal(m.nb_cell))
    f.assemble_poisson(torch.as_tensor(k, device="cuda"))
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_TRI3, coeff=k), "coefficient")
    rhs = torch.zeros(m.nb_node, dtype=torch.float64, device="cuda")
    f.rhs_constant_source(-5.5, rhs)
    ptr, nc, _ = O.node_cell(m.nb_node, m.cells)
    assert_bit_exact(rhs.cpu().numpy(), O.rhs_constant_source(2, m.coords, m.cells, ptr, nc, -5.5), "source")


MAKE = {"quad": meshgen.unit_square_quad, "tet": meshgen.unit_cube_tet, "hex": meshgen.unit_cube_hex}


@pytest.mark.parametrize("n,jitter,case", CASES)
def test_quadrangles_over_the_operand_ranges(own_ctx, n, jitter, case):
    m = moved_mesh(meshgen.unit_square_quad, 3 * n, jitter, case)
    f = build_format(own_ctx, m)
    f.assemble_poisson()
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_QUAD4), "quadrangles")
    k = np.exp(np.random.default_rng(0).standard_normal(m.nb_cell))
    f.assemble_poisson(torch.as_tensor(k, device="cuda"))
    assert_bit_exact(f.values.cpu().numpy(), oracle_values(m, O.POISSON_QUAD4, coeff=k), "coefficient")


@pytest.mark.parametrize("qdot", [-5.5, 0.0, 2.0 ** 245, 2.0 ** -243])
@pytest.mark.parametrize("kind", list(MAKE))
@pytest.mark.parametrize("n,jitter,case", CASES)
def test_sources_over_the_operand_ranges(own_ctx, kind, n, jitter, case, qdot):
    m = moved_mesh(MAKE[kind], n, jitter, case)
    f = build_format(own_ctx, m)
    rhs = torch.zeros(m.nb_node, dtype=torch.float64, device="cuda")
    f.rhs_constant_source(qdot, rhs)
    ptr, nc, _ = O.node_cell(m.nb_node, m.cells)
    fn = O.rhs_constant_source if kind == "tet" else O.rhs_constant_source_q1
    assert_bit_exact(rhs.cpu().numpy(), fn(m.dim, m.coords, m.cells, ptr, nc, qdot), "source")


def test_hexahedra_into_a_buffer_at_an_odd_double(own_ctx):
    m = meshgen.unit_cube_hex(3, jitter=0.15, seed=1)
    f = build_format(own_ctx, m)
    ke = torch.zeros(2 * f.element_buffer_size() + 2, dtype=torch.float64, device="cuda")
    size = f.element_buffer_size()
    f.element_matrices(ke[:size])
    f.element_matrices(ke[size + 1:2 * size + 1])
    assert torch.equal(ke[:size], ke[size + 1:2 * size + 1]) and float(ke[size]) == 0.0

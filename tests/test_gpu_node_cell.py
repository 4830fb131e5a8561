"""Node -> cell lists of nodes in more cells than a bucket of the build holds
(half again the mesh's average), and the rows built on them, against the CPU
oracle: bit-exact."""
import numpy as np
import pytest

from arcanefem_gb300 import fem, meshgen
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(ctx, dim, coords, cells):
    f = fem.BSRFormat(ctx, fem.Mesh.from_host(dim, coords, cells))
    f.initialize(1, True, fem.COLS_ASCENDING)
    f.compute_sparsity()
    ptr, nc, loc = O.node_cell(len(coords), cells)
    assert np.array_equal(f.nc_ptr.cpu().numpy(), ptr)
    assert np.array_equal(f.nc_cell.cpu().numpy(), nc)
    assert np.array_equal(f.nc_local.cpu().numpy(), loc)
    rp, cols = O.sparsity(len(coords), cells)
    assert np.array_equal(f.row_ptr.cpu().numpy(), rp)
    assert np.array_equal(f.cols.cpu().numpy(), cols)


# a node in k cells of an ordinary mesh: buckets of 16 keys (triangles) and 32 (tetrahedra), sorts of up to 32
@pytest.mark.parametrize("k", [1, 15, 16, 17, 31, 32, 33, 34, 200])
@pytest.mark.parametrize("kind", ["tri", "tet"])
def test_hub(cuda_ctx, kind, k):
    m = meshgen.unit_square_tri(20, seed=1) if kind == "tri" else meshgen.unit_cube_tet(12, seed=1)
    rng = np.random.default_rng(k)
    hub, npc = m.nb_node, m.cells.shape[1]
    ring = hub + npc - 2 + np.arange(k + 1)          # hub (and for tetrahedra the other end of its edge), then the ring
    fan = np.stack([np.full(k, hub + j) for j in range(npc - 2)] + [ring[:-1], ring[1:]], axis=1)
    cells = np.concatenate([m.cells, fan]).astype(np.int32)
    cells = np.stack([np.roll(c, s) for c, s in zip(cells, rng.integers(0, npc, len(cells)))]).astype(np.int32)
    coords = np.concatenate([m.coords, rng.random((npc - 2 + k + 1, 3))])
    check(cuda_ctx, m.dim, coords, cells[rng.permutation(len(cells))])


# every node in more cells than the largest bucket
@pytest.mark.parametrize("npc,nodes,nb_cell", [(3, 30, 2000), (4, 5, 400), (3, 3, 1)])
def test_all_nodes_spill(cuda_ctx, npc, nodes, nb_cell):
    rng = np.random.default_rng(nodes)
    cells = np.stack([rng.permutation(nodes)[:npc] for _ in range(nb_cell)]).astype(np.int32)
    check(cuda_ctx, 2 if npc == 3 else 3, rng.random((nodes, 3)), cells)

"""The work that programs hand to arcanefem_gb300, as cases for a timing harness.

Each case is one stage of a finite-element program, called through the
package's public classes the way `examples/poisson_msh.py`, `learned.setup`
and `batch.Batch` call them:

* module     -- the Poisson module's whole run on a mesh in hand: connectivity,
                sparsity, assembly, source, boundary condition, CG solve;
* structure  -- node-to-cell connectivity and the sparsity of a new mesh;
* assemble   -- the matrix, the right-hand side and the Dirichlet elimination
                of one time step on a mesh whose structure is kept;
* host       -- the matrix of one step from host coordinates to host values;
* solve      -- the Krylov solve of an assembled system;
* learned    -- the flexible CG with the learned V-cycle preconditioner;
* train      -- loss and gradients of that preconditioner for a batch of pairs;
* batch      -- many uneven 2D problems with 4 right-hand sides in one launch.

Meshes are the jittered structured ones of `arcanefem_gb300.meshgen`, made on
the GPU, each cell starting at a node of its own as in a mesh file; numbering
"grid" keeps their lexicographic ids, "shuffled" renumbers nodes and cells at
random, the worst an unstructured mesh file brings.
Solves run to a relative residual of 1e-10, `examples/poisson_msh.py`'s.
"""
import math

import numpy as np
import torch

from arcanefem_gb300 import batch, fem, learned, meshgen

NPC = {"tri": 3, "tet": 4, "quad": 4, "hexa": 8}
DIM = {"tri": 2, "tet": 3, "quad": 2, "hexa": 3}
PER_GRID_CELL = {"tri": 2, "tet": 6, "quad": 1, "hexa": 1}
ROW = {"tri": 7.0, "tet": 15.0, "quad": 9.0, "hexa": 27.0}   # entries of an interior row
YOUNG, POISSON = 21.0e5, 0.28                                # the elasticity bar of the tests' golden cases
SOURCE, FORCE, FIXED = -1.0, (0.0, 0.0, -1.0), 0.5
RTOL = 1e-10


def listed():
    return [
        # a 2D sanity run, as in the module's own test inputs: all latency and launches
        {"name": "module-tri-24", "kind": "module", "mesh": "tri", "n": 24, "numbering": "grid"},
        # the structure of the 128^3 Poisson benchmark mesh
        {"name": "structure-tet-128", "kind": "structure", "mesh": "tet", "n": 128, "dof": 1, "numbering": "grid"},
        # a 2D mesh as a mesh file may number it
        {"name": "structure-tri-701-shuffled", "kind": "structure", "mesh": "tri", "n": 701, "dof": 1,
         "numbering": "shuffled"},
        # the Poisson benchmark's matrix, reassembled in a time step
        {"name": "assemble-tet-128", "kind": "assemble", "mesh": "tet", "n": 128, "dof": 1, "numbering": "grid"},
        # a 3-DoF time step, CSR-compatible layout
        {"name": "assemble-elasticity-63", "kind": "assemble", "mesh": "tet", "n": 63, "dof": 3, "numbering": "grid"},
        # a CPU-side program that uploads moved coordinates and takes the matrix back
        {"name": "host-hexa-72", "kind": "host", "mesh": "hexa", "n": 72, "numbering": "grid"},
        # the 256^2 Poisson configuration's solve: small systems, many iterations
        {"name": "solve-tri-256", "kind": "solve", "mesh": "tri", "n": 256, "dof": 1, "precision": "fp64",
         "numbering": "grid"},
        # the 128^3 Poisson benchmark's solve
        {"name": "solve-tet-128", "kind": "solve", "mesh": "tet", "n": 128, "dof": 1, "precision": "fp64",
         "numbering": "grid"},
        # a 3-DoF solve in mixed precision (the 3x3-block SpMV)
        {"name": "solve-elasticity-40-mixed", "kind": "solve", "mesh": "tet", "n": 40, "dof": 3,
         "precision": "mixed", "numbering": "grid"},
        # the learned-preconditioner configuration (513^2 nodes)
        {"name": "learned-512", "kind": "learned", "n": 512, "levels": 9, "layers": 6},
        # one training batch of that network on a smaller grid
        {"name": "train-256-16", "kind": "train", "n": 256, "levels": 8, "layers": 6, "pairs": 16},
        # uneven small problems solved together
        {"name": "batch-12", "kind": "batch", "count": 12, "nmin": 64, "nmax": 384, "sizes_seed": 2024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["module", "structure", "structure", "assemble", "assemble", "host", "solve", "solve",
                       "learned", "train", "batch"])
    numbering = rng.choice(["grid", "grid", "shuffled"])
    mesh = rng.choice(["tri", "tet", "quad", "hexa"])
    if kind == "module":
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 16, 200) if DIM[mesh] == 2 else _log_int(rng, 6, 30),
                "numbering": numbering}
    if kind in ("structure", "assemble"):
        dof = 3 if mesh == "tet" and rng.random() < 0.4 else 1
        hi = {"tri": 1200, "quad": 1200, "tet": 128 if dof == 1 else 63, "hexa": 90}[mesh]
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 24 if DIM[mesh] == 2 else 8, hi), "dof": dof,
                "numbering": numbering}
    if kind == "host":
        hi = {"tri": 1000, "quad": 1000, "tet": 96, "hexa": 72}[mesh]
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 64 if DIM[mesh] == 2 else 12, hi),
                "numbering": "grid"}
    if kind == "solve":
        dof = 3 if mesh == "tet" and rng.random() < 0.4 else 1
        hi = {"tri": 600, "quad": 600, "tet": 110 if dof == 1 else 40, "hexa": 90}[mesh]
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 32 if DIM[mesh] == 2 else 8, hi), "dof": dof,
                "precision": rng.choice(["fp64", "fp64", "mixed"]), "numbering": numbering}
    if kind == "learned":
        levels = rng.choice([6, 7, 8])
        step = 1 << (levels - 1)
        return {"kind": kind, "n": step * rng.randint(2, max(2, 512 // step)), "levels": levels,
                "layers": rng.randint(4, 6)}
    if kind == "train":
        levels = rng.choice([5, 6, 7])
        step = 1 << (levels - 1)
        return {"kind": kind, "n": step * rng.randint(2, max(2, 256 // step)), "levels": levels,
                "layers": rng.randint(4, 5), "pairs": rng.choice([1, 4, 8, 16])}
    return {"kind": "batch", "count": rng.randint(2, 12), "nmin": rng.randint(24, 100), "nmax": rng.randint(128, 384),
            "sizes_seed": rng.randint(1, 10000)}


# ---------------------------------------------------------------------------
# Inputs

def _mesh(kind, n, seed, numbering):
    """(fem.Mesh, boundary node ids): the jittered structured mesh of meshgen, made on the GPU."""
    dim, m, h = DIM[kind], n + 1, 1.0 / n
    gen = torch.Generator(device="cuda").manual_seed(seed)
    one = {"tri": meshgen.unit_square_tri, "quad": meshgen.unit_square_quad, "tet": meshgen.unit_cube_tet,
           "hexa": meshgen.unit_cube_hex}[kind](1, jitter=0.0)
    ax = torch.arange(m, device="cuda")
    grid = torch.meshgrid(*([ax] * dim), indexing="ij")[::-1]      # grid[0] is the fastest index
    idx = torch.stack([g.reshape(-1) for g in grid], 1)            # [N, dim]
    coords = torch.zeros((m ** dim, 3), dtype=torch.float64, device="cuda")
    coords[:, :dim] = idx.double() * h
    bnd = ((idx == 0) | (idx == n)).any(1)
    move = (torch.rand((m ** dim, dim), generator=gen, dtype=torch.float64, device="cuda") * 2 - 1)
    coords[:, :dim] += move * ((0.2 if dim == 2 else 0.15) * h) * (~bnd)[:, None]
    cx = torch.arange(n, device="cuda")
    cgrid = torch.meshgrid(*([cx] * dim), indexing="ij")[::-1]
    base = sum(g.reshape(-1) * m ** d for d, g in enumerate(cgrid))
    corner = torch.as_tensor([sum(((c >> d) & 1) * m ** d for d in range(dim)) for c in range(1 << dim)], device="cuda")
    template = corner[torch.as_tensor(one.cells.astype(np.int64), device="cuda")]
    cells = (base[:, None, None] + template[None]).reshape(-1, NPC[kind]).to(torch.int32)
    turn = torch.randint(0, 3, (cells.shape[0],), generator=gen, device="cuda")
    cells = cells[torch.arange(cells.shape[0], device="cuda")[:, None], _turns(kind)[turn]]
    if numbering == "shuffled":
        perm = torch.randperm(m ** dim, generator=gen, device="cuda")
        at = int(torch.nonzero(perm == 0))
        perm[at] = perm[0].clone()
        perm[0] = 0                                                # node 0 stays a corner, on the boundary
        moved = torch.empty_like(coords)
        moved[perm] = coords
        coords = moved
        flag = torch.empty_like(bnd)
        flag[perm] = bnd
        bnd = flag
        cells = perm[cells.long()].to(torch.int32)
        cells = cells[torch.randperm(cells.shape[0], generator=gen, device="cuda")]
    return fem.Mesh(dim, coords.contiguous(), cells.contiguous()), torch.nonzero(bnd).reshape(-1).to(torch.int32)


def _turns(kind):
    """Three orders of a cell's nodes that keep its orientation: a mesh file starts a cell at any of its nodes."""
    one = {"tri": [[0, 1, 2], [1, 2, 0], [2, 0, 1]], "tet": [[0, 1, 2, 3], [0, 2, 3, 1], [1, 2, 0, 3]],
           "quad": [[0, 1, 2, 3], [1, 2, 3, 0], [3, 0, 1, 2]],
           "hexa": [[0, 1, 2, 3, 4, 5, 6, 7], [1, 2, 3, 0, 5, 6, 7, 4], [3, 0, 1, 2, 7, 4, 5, 6]]}[kind]
    return torch.as_tensor(one, device="cuda")


def _format(ctx, mesh, dof):
    fmt = fem.BSRFormat(ctx, mesh)
    fmt.initialize(dof)
    fmt.compute_sparsity()
    return fmt


def _assemble(fmt):
    if fmt.nb_dof == 3:
        fmt.assemble_elasticity(*fem.lame(YOUNG, POISSON))
    else:
        fmt.assemble_poisson()


def _rhs(fmt, rhs):
    if fmt.nb_dof == 3:
        rhs.zero_()
        fmt.rhs_body_force(FORCE, rhs)
    else:
        fmt.rhs_constant_source(SOURCE, rhs)


def _fixed(case, mesh, bnd):
    """The Dirichlet nodes: the whole boundary, or the face x = 0 of an elastic body (node 0 is on it)."""
    return bnd if case.get("dof", 1) == 1 else bnd[mesh.coords[bnd.long(), 0] < 1e-9]


def _boundary(ls, fixed, dof, value):
    for k in range(dof):
        ls.apply_dirichlet_elimination(fem.ELIMINATE_ROW_COLUMN, fixed, dof, k, value)
    ls.apply_matrix_transformation()
    ls.apply_rhs_transformation()


def _diffusion(case, seed):
    """The learned-preconditioner problem and network of learned.setup, with small random edge heads."""
    ctx = fem.Context()
    prob = learned.DiffusionProblem(ctx, n=case["n"], seed=seed)
    hier = learned.Hierarchy(case["n"], case["levels"], prob.row_ptr, prob.cols)
    net = learned.MPNN(ctx, hier, layers=case["layers"], max_batch=case.get("pairs", 1))
    net.set_params(net.init_params(seed, edge_scale=0.02))
    net.set_operator(prob.row_ptr, prob.cols, prob.values)
    return ctx, prob, hier, net


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ctx = fem.Context()
        sizes = batch.instance_sizes(case["count"], case["nmin"], case["nmax"], case["sizes_seed"])
        return {"kind": kind, "ctx": ctx, "batch": batch.Batch(ctx, sizes, seed=seed, jitter=0.2),
                "options": fem.solver_options(rtol=RTOL, inner_rtol=0.1, max_iter=20000)}
    if kind == "learned":
        ctx, prob, hier, net = _diffusion(case, seed)
        b = prob.rhs(np.random.default_rng(seed + 5))
        return {"kind": kind, "ctx": ctx, "prob": prob, "hier": hier, "net": net, "b": b,
                "options": fem.solver_options(rtol=RTOL, max_iter=500)}
    if kind == "train":
        ctx, prob, hier, net = _diffusion(case, seed)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        e = torch.randn((case["pairs"], prob.mesh.nb_node), generator=gen, dtype=torch.float64, device="cuda")
        e = e * prob.interior
        dinv = 1.0 / prob.lumped
        for _ in range(6):                       # smooth the errors a little, as a few solver steps do
            r = torch.stack([prob.apply(v.contiguous()) for v in e])
            e = e - 0.02 * r * dinv / (dinv.max() * 8.0) * prob.interior
        r = torch.stack([prob.apply(v.contiguous()) for v in e])
        return {"kind": kind, "ctx": ctx, "prob": prob, "hier": hier, "net": net, "r": r.float().contiguous(),
                "e": e.float().contiguous()}
    mesh, bnd = _mesh(case["mesh"], case["n"], seed, case["numbering"])
    s = {"kind": kind, "ctx": fem.Context(), "mesh": mesh, "dof": case.get("dof", 1)}
    s["fixed"] = _fixed(case, mesh, bnd)
    if kind == "module":
        s["options"] = fem.solver_options(rtol=RTOL, max_iter=100000)
    if kind in ("module", "structure"):
        return s
    fmt = s["fmt"] = _format(s["ctx"], mesh, s["dof"])
    if kind == "host":
        s["coords"] = mesh.coords.cpu().pin_memory()
        s["ke"] = torch.empty(fmt.element_buffer_size(), dtype=torch.float64, device="cuda")
        s["values"] = torch.empty(fmt.values.numel(), dtype=torch.float64).pin_memory()
        return s
    ls = s["ls"] = fem.DoFLinearSystem(s["ctx"], mesh.nb_node * s["dof"])
    fmt.to_linear_system(ls)
    if kind == "solve":
        _assemble(fmt)
        _rhs(fmt, ls.rhs_variable())
        _boundary(ls, s["fixed"], s["dof"], 0.0)
        mixed = case["precision"] == "mixed"
        s["options"] = fem.solver_options(rtol=RTOL, max_iter=100000,
                                          precision=fem.PRECISION_MIXED if mixed else fem.PRECISION_FP64)
    return s


# ---------------------------------------------------------------------------
# One pass.  The linear system's variables are views of its own memory: they are copied out, as a
# program does that keeps them after the system.

def run(s):
    kind = s["kind"]
    if kind == "module":
        fmt = _format(s["ctx"], s["mesh"], 1)
        fmt.assemble_poisson()
        ls = fem.DoFLinearSystem(s["ctx"], s["mesh"].nb_node)
        fmt.to_linear_system(ls)
        fmt.rhs_constant_source(SOURCE, ls.rhs_variable())
        ls.apply_dirichlet_elimination(fem.ELIMINATE_ROW_COLUMN, s["fixed"], 1, 0, 0.0)
        ls.apply_linear_system_transformation_and_solve(s["options"])
        u = ls.solution_variable().clone()
        ls.close()
        return u
    if kind == "structure":
        fmt = _format(s["ctx"], s["mesh"], s["dof"])
        rp, cols, _ = fmt.to_csr()
        return {"nc_ptr": fmt.nc_ptr, "nc_cell": fmt.nc_cell, "nc_local": fmt.nc_local, "nc_inverse": fmt.nc_inverse,
                "nc_slot": fmt.nc_slot, "brow_ptr": fmt.row_ptr, "bcols": fmt.cols, "row_ptr": rp, "cols": cols}
    if kind == "assemble":
        _assemble(s["fmt"])
        _rhs(s["fmt"], s["ls"].rhs_variable())
        _boundary(s["ls"], s["fixed"], s["dof"], FIXED)
        return {"values": s["fmt"].values, "rhs": s["ls"].rhs_variable().clone()}
    if kind == "host":
        s["fmt"].assemble_to_host(s["ke"], s["values"], coords_h=s["coords"])
        return s["values"]
    if kind == "solve":
        s["ls"].solution_variable().zero_()
        s["ls"].solve(s["options"])
        return s["ls"].solution_variable().clone()
    if kind == "learned":
        p = s["prob"]
        x = torch.zeros_like(s["b"])
        s["net"].fcg(p.row_ptr, p.cols, p.values, s["b"], x, s["options"])
        return x
    if kind == "train":
        grad, loss = s["net"].gradients(s["r"], s["e"])
        return {"grad": grad, "loss": loss}
    s["batch"].solve(s["options"])
    return {"x": list(s["batch"].x), "rhs": list(s["batch"].rhs)}


# ---------------------------------------------------------------------------
# What a pass cannot do without

def _counts(case):
    kind, n = case["mesh"], case["n"]
    nodes, cells = (n + 1) ** DIM[kind], PER_GRID_CELL[kind] * n ** DIM[kind]
    return nodes, cells, NPC[kind], ROW[kind] * nodes


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = batch.instance_sizes(case["count"], case["nmin"], case["nmax"], case["sizes_seed"])
        nodes = sum((n + 1.0) ** 2 for n in sizes)
        # about 4 n Jacobi CG iterations of 4 right-hand sides each; mesh and structure in, values, rhs and x out
        flops = sum(4.0 * n * 4 * (n + 1.0) ** 2 * (2 * 7 + 10) for n in sizes)
        return {"bytes": nodes * (24 + 2 * 12 + 7 * 4 + 7 * 8 + 2 * 32), "flops": flops}
    if kind in ("learned", "train"):
        n0 = (case["n"] + 1.0) ** 2
        if kind == "learned":   # about 13 iterations: A p, two smoothings and residuals a level, 4/3 levels
            return {"bytes": n0 * (7 * 12 + 2 * 8), "flops": 13 * n0 * (2 * 7 + 4 / 3 * 60)}
        flops = 3 * 4 / 3 * n0 * 2 * 2 * 64 * 64 + 3 * case["pairs"] * 4 / 3 * n0 * 60
        return {"bytes": n0 * (7 * 12 + 8 * case["pairs"]), "flops": flops}
    nodes, cells, npc, nnz = _counts(case)
    dof = case.get("dof", 1)
    inc = cells * npc
    structure = 4 * nodes + 4 * inc + inc + 4 * inc + 4 * nodes + 4 * nnz + inc * npc
    element = {"tri": 60, "tet": 230, "quad": 700, "hexa": 4700}[case["mesh"]] if dof == 1 else 640
    if kind == "structure":
        return {"bytes": 4 * inc + structure + (8 * nnz if dof == 1 else 72 * nnz + 36 * nnz + 12 * nodes), "flops": 0}
    if kind in ("assemble", "host"):
        rows = 0 if kind == "host" else (5 * nnz if dof == 1 else 45 * nnz) + 8 * dof * nodes
        return {"bytes": 24 * nodes + 4 * inc + 8 * dof * dof * nnz + rows, "flops": cells * element}
    per_pass = 2 * dof * dof * nnz + 12 * dof * nodes
    iters = (4.3 if DIM[case["mesh"]] == 2 else 5.5) * case["n"] * (1 if dof == 1 else 4)
    if kind == "module":
        return {"bytes": 24 * nodes + 4 * inc + structure + 8 * nnz + 16 * nodes,
                "flops": cells * element + iters * per_pass}
    return {"bytes": 12 * dof * dof * nnz + 16 * dof * nodes, "flops": iters * per_pass}


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch

def _shape_gradients(x, kind):
    """[(gradients [C, npc, dim], weight [C], shape values [npc])] of the cells with corners x [C, npc, dim]."""
    npc, dim = x.shape[1], x.shape[2]
    if kind in ("tri", "tet"):
        e = x[:, 1:] - x[:, :1]
        if dim == 2:
            det = e[:, 0, 0] * e[:, 1, 1] - e[:, 0, 1] * e[:, 1, 0]
            g = torch.stack([torch.stack([e[:, 1, 1], -e[:, 1, 0]], 1), torch.stack([-e[:, 0, 1], e[:, 0, 0]], 1)], 1)
        else:
            c = [torch.linalg.cross(e[:, (k + 1) % 3], e[:, (k + 2) % 3]) for k in range(3)]
            det = (e[:, 0] * c[0]).sum(1)
            g = torch.stack(c, 1)
        g = g / det[:, None, None]
        return [(torch.cat([-g.sum(1, keepdim=True), g], 1), det.abs() / (2 if dim == 2 else 6), [1.0 / npc] * npc)]
    corners = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
    corners = [c[:dim] for c in corners[:npc]]
    a, points = 1.0 / math.sqrt(3.0), []
    for q in range(1 << dim):
        pt = [a if (q >> d) & 1 else -a for d in range(dim)]
        f = [[0.5 * (1 + c[d] * pt[d]) for d in range(dim)] for c in corners]
        dn = [[0.5 * c[d] * math.prod(f[i][o] for o in range(dim) if o != d) for d in range(dim)]
              for i, c in enumerate(corners)]
        dn = torch.tensor(dn, dtype=torch.float64, device=x.device)
        jac = torch.einsum("nd,cne->cde", dn, x)
        points.append((torch.einsum("ced,nd->cne", torch.linalg.inv(jac), dn), torch.linalg.det(jac).abs(),
                       [math.prod(v) for v in f]))
    return points


def _system(kind, coords, cells, dof=1, coeff=None, chunk=1 << 19):
    """(row pointers, columns, block values [nnz, dof, dof], load weights [N]) of the assembled matrix, columns ascending."""
    n, npc, dim = coords.shape[0], cells.shape[1], DIM[kind]
    cl = cells.long()
    keys = torch.empty(0, dtype=torch.int64, device=coords.device)
    step = max(1, (1 << 26) // (npc * npc))
    for c0 in range(0, cl.shape[0], step):
        c = cl[c0:c0 + step]
        keys = torch.unique(torch.cat([keys, (c[:, :, None] * n + c[:, None, :]).reshape(-1)]))
    rows, cols = keys // n, keys % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device=coords.device)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    values = torch.zeros((keys.numel(), dof, dof), dtype=torch.float64, device=coords.device)
    load = torch.zeros(n, dtype=torch.float64, device=coords.device)
    lam, mu = fem.lame(YOUNG, POISSON)
    for c0 in range(0, cl.shape[0], chunk):
        c = cl[c0:c0 + chunk]
        at = torch.searchsorted(keys, (c[:, :, None] * n + c[:, None, :]).reshape(-1))
        k = 0.0
        for g, w, shape in _shape_gradients(coords[c][:, :, :dim], kind):
            dot = torch.einsum("cid,ckd->cik", g, g)
            if dof == 1:
                k = k + (dot * w[:, None, None])[..., None, None]
            else:
                outer = torch.einsum("cia,ckb->cikab", g, g)
                eye = torch.eye(3, dtype=torch.float64, device=g.device)
                k = k + (lam * outer + mu * outer.transpose(3, 4) + mu * dot[..., None, None] * eye) * w[:, None, None, None, None]
            for i in range(npc):
                load.index_add_(0, c[:, i], w * shape[i])
        if coeff is not None:
            k = k * coeff[c0:c0 + chunk, None, None, None, None]
        values.index_add_(0, at, k.reshape(-1, dof, dof))
    return rp, rows, cols, values, load


def _eliminated(rows, cols, values, rhs, fixed, value):
    """Row-column elimination of the nodes in the mask `fixed`; as the reference, entries of column 0 stay."""
    dof = values.shape[1]
    hit = fixed[cols] & ~fixed[rows]
    rhs = rhs.index_add(0, rows[hit], -(values[hit] * value).sum(2)) if value else rhs.clone()
    gone = fixed[rows] | fixed[cols]
    eye = torch.eye(dof, dtype=torch.float64, device=values.device)
    keep0 = torch.zeros((values.shape[0], dof, dof), dtype=torch.bool, device=values.device)
    keep0[cols == 0, :, 0] = True
    ident = torch.where((rows == cols)[:, None, None], eye, torch.zeros_like(eye))
    values = torch.where(gone[:, None, None] & ~keep0, ident, values)
    rhs[fixed] = value
    return values, rhs


def _scalar_values(rp, rows, values):
    """Block values [nnzb, b, b] in the order of the scalar CSR rows."""
    b = values.shape[1]
    if b == 1:
        return values.reshape(-1)
    length = (rp[1:] - rp[:-1])[rows]
    x = torch.arange(rows.numel(), device=rows.device) - rp[rows]
    out = torch.empty(values.numel(), dtype=torch.float64, device=values.device)
    for i in range(b):
        for j in range(b):
            out[9 * rp[rows] + 3 * (x + i * length) + j] = values[:, i, j]
    return out


def _solution(rows, cols, values, rhs, fixed):
    """A x = rhs (x given on the fixed nodes, whose columns are moved over) by Jacobi CG on [N b, k], to rounding."""
    n, b = fixed.numel(), values.shape[1]
    free = ~fixed
    inner = free[rows] & free[cols]
    r, c, v = rows[inner], cols[inner], values[inner]
    comp = torch.arange(b, device=rows.device)
    sr = (r[:, None, None] * b + comp[:, None]).expand(-1, b, b).reshape(-1)
    sc = (c[:, None, None] * b + comp[None, :]).expand(-1, b, b).reshape(-1)
    order = torch.argsort(sr * (n * b) + sc)
    ptr = torch.zeros(n * b + 1, dtype=torch.int64, device=rows.device)
    ptr[1:] = torch.cumsum(torch.bincount(sr, minlength=n * b), 0)
    A = torch.sparse_csr_tensor(ptr, sc[order], v.reshape(-1)[order], size=(n * b, n * b))
    d = torch.zeros(n * b, dtype=torch.float64, device=rows.device)
    on = sr == sc
    d[sr[on]] = v.reshape(-1)[on]
    dinv = torch.where(d != 0, 1.0 / torch.where(d != 0, d, torch.ones_like(d)), torch.zeros_like(d))[:, None]
    mask = free.repeat_interleave(b)[:, None].double()
    f = rhs.reshape(n * b, -1) * mask
    x = torch.zeros_like(f)
    res, stop = f.clone(), 1e-14 * torch.linalg.norm(f, dim=0)
    for _ in range(3):                                             # restarts from the true residual
        z = dinv * res
        p, rz = z.clone(), (res * z).sum(0)
        for k in range(40000):
            q = A @ p
            alpha = rz / torch.clamp((p * q).sum(0), min=1e-300)
            x += alpha * p
            res -= alpha * q
            if k % 50 == 49 and bool((torch.linalg.norm(res, dim=0) <= stop).all()):
                break
            z = dinv * res
            new = (res * z).sum(0)
            p = z + (new / torch.clamp(rz, min=1e-300)) * p
            rz = new
        res = f - A @ x
    return x + (1 - mask) * rhs.reshape(n * b, -1)


def _mask(n, nodes):
    m = torch.zeros(n, dtype=torch.bool, device="cuda")
    m[nodes.long()] = True
    return m


def exact(case, seed):
    kind = case["kind"]
    if kind in ("structure", "train"):   # whole numbers; a network that is defined in bfloat16
        return None
    if kind == "learned":
        ctx = fem.Context()
        prob = learned.DiffusionProblem(ctx, n=case["n"], seed=seed)
        b = prob.rhs(np.random.default_rng(seed + 5))
        coeff = torch.as_tensor(prob.k, device="cuda")
        _, rows, cols, values, _ = _system("tri", prob.fmt.mesh.coords, prob.fmt.mesh.cells, coeff=coeff)
        return _solution(rows, cols, values, b, _mask(b.numel(), prob.boundary)).reshape(-1)
    if kind == "batch":
        ctx = fem.Context()
        sizes = batch.instance_sizes(case["count"], case["nmin"], case["nmax"], case["sizes_seed"])
        made = batch.Batch(ctx, sizes, seed=seed, jitter=0.2)
        xs, bs = [], []
        for fmt, src, dirichlet in zip(made.fmts, made.sources, made.dirichlet):
            xy = fmt.mesh.coords
            _, rows, cols, values, load = _system("tri", xy, fmt.mesh.cells)
            s = src.double()                                       # [4][8]: amplitude, centre, width
            d2 = (xy[:, None, None, 0] - s[None, :, :, 1]) ** 2 + (xy[:, None, None, 1] - s[None, :, :, 2]) ** 2
            f = (s[None, :, :, 0] * torch.exp(-d2 / (2 * s[None, :, :, 3] ** 2))).sum(2)
            fixed = dirichlet.bool()
            b = load[:, None] * f * (~fixed)[:, None]
            bs.append(b)
            xs.append(_solution(rows, cols, values, b, fixed))
        return {"x": xs, "rhs": bs}
    mesh, bnd = _mesh(case["mesh"], case["n"], seed, case["numbering"])
    dof = case.get("dof", 1)
    rp, rows, cols, values, load = _system(case["mesh"], mesh.coords, mesh.cells, dof)
    if kind == "host":
        return _scalar_values(rp, rows, values)
    force = [SOURCE] if dof == 1 else FORCE
    rhs = torch.stack([f * load for f in force], 1)
    fixed = _mask(mesh.nb_node, _fixed(case, mesh, bnd))
    if kind == "assemble":
        values, rhs = _eliminated(rows, cols, values, rhs, fixed, FIXED)
        return {"values": _scalar_values(rp, rows, values), "rhs": rhs.reshape(-1)}
    rhs[fixed] = 0.0
    return _solution(rows, cols, values, rhs, fixed).reshape(-1)

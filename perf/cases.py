"""Performance cases of the transport framework: what a user of it runs, by call.

A simulation ingests a mesh once (GPUSparseAssembler), then steps: assemble the operator
and right-hand side, apply or solve it, advance the level set.  It does so through the
reference-shaped calls (solve_transport, CeedDiffusionMassOp.apply), through the step
drivers (PlainTransport, BatchedTransport, GyroidStep, MeshBatch) or with the learned
initial guess (WarmStartMLP).  Each listed case is one of those calls; `draw` gives more of
the same calls on boxes of other sizes, square or not, with the other options.

Meshes are jittered Kuhn-split boxes of nx x ny x nz cells, as in the repository's
configurations (16^3, 48^3, 64^3, uneven batches of 8..40 per side), and coefficients and
fields follow the same distributions: De = D exp(0.3 N(0,1)), u ~ U(0,1), dt 0.02 or 0.05.
Solves run to 1e-10 (1e-12 with Dirichlet rows, whose large entries of b weaken the relative
rule), tight enough that two correct solvers agree to about 1e-11; the mixed-precision step
then refreshes its residual every factor 100 (delta 0.01).
"""
import math
import os
import sys
import types

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "dissolve-2.0_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

D_S, K_S = (1.0, 1.0, 2.6), (0.5, 0.0, 0.2)  # O2, Cl-, OH-
PERMS = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))


# ------------------------------------------------------------------ cases
def listed():
    return [
        # ingest of a mesh up to its first assembled operator: once per mesh or remesh
        dict(name="setup_64", kind="setup", nx=64, ny=64, nz=64, jitter=0.2),
        # the FP64 backward-Euler operator of one species, per-cell coefficients, lumped mass
        dict(name="assemble_64", kind="assemble", nx=64, ny=64, nz=64, jitter=0.2, lumped=True,
             alpha=True, bc=False, vertex_coef=False),
        # the right-hand side with a source, consistent mass, on a ragged box
        dict(name="rhs_57x64x71", kind="rhs", nx=57, ny=64, nz=71, jitter=0.2, lumped=False,
             source=True, bc=True),
        # the matrix-free operator on one field (a Krylov product of the MatShell path)
        dict(name="apply_64", kind="apply", nx=64, ny=64, nz=64, jitter=0.2),
        # the smallest call: one species' solve_transport on host arrays with Dirichlet rows
        dict(name="transport_16", kind="transport", nx=16, ny=16, nz=16, jitter=0.15,
             rtol=1e-12),
        # the plain FP64 step, one species after the other, at the headline size
        dict(name="plain_64", kind="plain", nx=64, ny=64, nz=64, jitter=0.2, species=3,
             rtol=1e-10),
        # the fast three-species step at the headline size, guess projected on the history
        dict(name="step_64", kind="step", nx=64, ny=64, nz=64, jitter=0.2, species=3,
             fp32=True, guess="project", host=False, rtol=1e-10),
        # the same step end to end through pinned host buffers on a small ragged mesh
        dict(name="step_host_23", kind="step", nx=23, ny=20, nz=26, jitter=0.2, species=3,
             fp32=True, guess="previous", host=True, rtol=1e-10),
        # the coupled gyroid step: interface reaction, three species, level-set advance
        dict(name="gyroid_48", kind="gyroid", nx=48, ny=48, nz=48, jitter=0.15, rtol=1e-10),
        # many uneven independent meshes stepped together
        dict(name="batch_64", kind="batch", meshes=64, n_min=8, n_max=40, rtol=1e-10),
        # the learned guess: inference over every vertex and species of the headline mesh ...
        dict(name="predict_64", kind="predict", verts=274625, species=3),
        # ... and one training gradient on the sampled rows
        dict(name="gradient_65536", kind="gradient", rows=65536),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        n = side(lo, hi)
        return dict(zip(("nx", "ny", "nz"),
                        (max(3, min(hi, int(round(n * rng.uniform(0.8, 1.25))))) for _ in "xyz")))

    kind = rng.choice(("setup", "assemble", "rhs", "apply", "transport", "plain", "step",
                       "gyroid", "batch", "predict", "gradient"))
    jitter = round(rng.uniform(0.05, 0.2), 3)
    coin = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "setup":
        return dict(kind=kind, jitter=jitter, **box(8, 64))
    if kind == "assemble":
        return dict(kind=kind, jitter=jitter, lumped=coin(), alpha=coin(), bc=coin(),
                    vertex_coef=coin(), **box(8, 72))
    if kind == "rhs":
        return dict(kind=kind, jitter=jitter, lumped=coin(), source=coin(), bc=coin(),
                    **box(8, 72))
    if kind == "apply":
        return dict(kind=kind, jitter=jitter, **box(8, 72))
    if kind == "transport":
        return dict(kind=kind, jitter=jitter, rtol=1e-12, **box(8, 32))
    if kind == "plain":
        return dict(kind=kind, jitter=jitter, species=rng.choice((1, 2, 3)), rtol=1e-10,
                    **box(10, 64))
    if kind == "step":
        return dict(kind=kind, jitter=jitter, species=rng.choice((2, 3, 3, 4)),
                    fp32=rng.random() < 0.75, guess=rng.choice(("previous", "project")),
                    host=coin(), rtol=1e-10, **box(10, 64))
    if kind == "gyroid":
        n = side(16, 56)
        return dict(kind=kind, jitter=jitter, nx=n, ny=n, nz=n, rtol=1e-10)
    if kind == "batch":
        return dict(kind=kind, meshes=side(4, 64), n_min=8, n_max=rng.randint(16, 40),
                    rtol=1e-10)
    if kind == "predict":
        return dict(kind=kind, verts=int(math.exp(rng.uniform(math.log(2e3), math.log(3e5)))),
                    species=rng.choice((1, 2, 3, 4)))
    return dict(kind=kind, rows=int(math.exp(rng.uniform(math.log(2e3), math.log(1.3e5)))))


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _rand(shape, g, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _normal(shape, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _box(nx, ny, nz, jitter, g, extent=1.0):
    """Jittered Kuhn-split box with cubic cells, vertex i + (nx+1)(j + (ny+1)k): coords (V, 3)
    and cells (n, 4) on the GPU.  The longest side has length `extent`."""
    h = extent / max(nx, ny, nz)
    ar = [torch.arange(n + 1, device="cuda") for n in (nx, ny, nz)]
    k, j, i = torch.meshgrid(ar[2], ar[1], ar[0], indexing="ij")
    ijk = torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)], 1)
    xyz = h * ijk.double()
    top = torch.tensor([nx, ny, nz], device="cuda")
    inner = ((ijk > 0) & (ijk < top)).all(1)
    xyz = xyz + inner[:, None] * _rand(xyz.shape, g, -jitter * h, jitter * h)
    k, j, i = torch.meshgrid(ar[2][:-1], ar[1][:-1], ar[0][:-1], indexing="ij")
    base = (i + (nx + 1) * (j + (ny + 1) * k)).reshape(-1)
    step = (1, nx + 1, (nx + 1) * (ny + 1))
    cells = torch.empty((base.numel(), 6, 4), dtype=torch.int32, device="cuda")
    for t, p in enumerate(PERMS):
        v = base
        cells[:, t, 0] = v
        for q in range(3):
            v = v + step[p[q]]
            cells[:, t, q + 1] = v
    return xyz, cells.reshape(-1, 4)


def _x0_face(xyz):
    return torch.nonzero(xyz[:, 0] == 0.0).reshape(-1).to(torch.int32)


def _mesh_inputs(case, seed, extent=1.0):
    g = _gen(seed)
    xyz, cells = _box(case["nx"], case["ny"], case["nz"], case["jitter"], g, extent)
    return g, xyz, cells


def _tetmesh(xyz, cells):
    from dissolve_tp.mesh import TetMesh
    return TetMesh(coords=xyz.cpu().numpy(), cells=cells.cpu().numpy())


def _assemble_inputs(case, seed):
    g, xyz, cells = _mesh_inputs(case, seed)
    n = xyz.shape[0] if case.get("vertex_coef") else cells.shape[0]
    De = torch.exp(0.3 * _normal(n, g))
    alpha = _rand(n, g, 0.0, 2.0) if case.get("alpha") else None
    bc = _x0_face(xyz) if case.get("bc") else None
    return xyz, cells, De, alpha, bc


def _rhs_inputs(case, seed):
    g, xyz, cells = _mesh_inputs(case, seed)
    V = xyz.shape[0]
    u = _rand(V, g)
    f = _rand(V, g, -1.0, 1.0) if case["source"] else None
    return xyz, cells, u, f, (_x0_face(xyz) if case["bc"] else None)


def _transport_inputs(case, seed):
    g, xyz, cells = _mesh_inputs(case, seed)
    V = xyz.shape[0]
    De, alpha, u = torch.exp(0.3 * _normal(V, g)), _rand(V, g, 0.0, 1.0), _rand(V, g)
    return xyz, cells, De, alpha, u, _x0_face(xyz)


def _step_inputs(case, seed):
    """Mesh, per-cell factor, two time levels (the newer one a smoothed move of the older)."""
    g, xyz, cells = _mesh_inputs(case, seed)
    S = case["species"]
    coef = torch.exp(0.3 * _normal(cells.shape[0], g))
    u0 = _rand((xyz.shape[0], S), g)
    u1 = 0.5 + 0.6 * (u0 - 0.5) + 0.1 * torch.sin(3.0 * xyz.sum(1, keepdim=True))
    return xyz, cells, coef, u0, u1


def _species(S):
    return (list(D_S) + [1.3])[:S], (list(K_S) + [0.1])[:S]


def _gyroid_inputs(case, seed):
    g, xyz, cells = _mesh_inputs(case, seed, 2.0 * math.pi)
    x, y, z = xyz.unbind(1)
    phi = (torch.sin(x) * torch.cos(y) + torch.sin(y) * torch.cos(z) +
           torch.sin(z) * torch.cos(x) - 0.3)
    coef = torch.exp(0.3 * _normal(cells.shape[0], g))
    return xyz, cells, phi, coef, _rand((xyz.shape[0], 3), g)


def _batch_inputs(case, seed):
    """Sizes belong to the case; jitter, D ~ LogUniform(0.1, 10), k ~ U(0, 1) to the seed."""
    sizes = np.random.default_rng(17 + case["meshes"]).integers(
        case["n_min"], case["n_max"] + 1, case["meshes"])
    rng = np.random.default_rng(seed)
    D = np.exp(rng.uniform(np.log(0.1), np.log(10.0), len(sizes)))
    k = rng.uniform(0.0, 1.0, len(sizes))
    g = _gen(seed)
    boxes = [_box(int(n), int(n), int(n), 0.2, g) for n in sizes]
    u = _rand(sum(b[0].shape[0] for b in boxes), g)
    return boxes, D, k, u


def _predict_inputs(case, seed):
    """State, history, level set and stiffness images of a learned step, as arrays."""
    g = _gen(seed)
    V, S = case["verts"], case["species"]
    ld = {1: 1, 2: 2, 3: 4, 4: 4}[S]

    def field(scale, shift=0.0):
        t = torch.zeros((V, ld), dtype=torch.float64, device="cuda")
        t[:, :S] = shift + scale * _normal((V, S), g)
        return t

    up = field(0.3, 0.5)
    un = up + field(0.05)
    nx = un + field(0.03)
    phi, ng = _normal(V, g), _rand(V, g, 0.5, 1.5)
    return up, un, nx, phi, ng, (field(0.2), field(0.02))


def _mlp(seed):
    """A network with weights of a trained one's size (all layers and biases non-zero)."""
    from dissolve_tp.mlp import WarmStartMLP
    mlp = WarmStartMLP(torch.device("cuda"), seed=3)
    mlp.params.copy_(_mlp_params(seed))
    return mlp


def _mlp_params(seed):
    g = _gen(seed, 7)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    W1 = r(64, 16) * math.sqrt(0.2)
    W1[:, 10:] = 0.0
    return torch.cat([W1.reshape(-1), 0.1 * r(64), (r(64, 64) * math.sqrt(2.0 / 64)).reshape(-1),
                      0.1 * r(64), r(64) * 0.1, 0.1 * r(1)])


def _gradient_fields(case, seed):
    """One training pair whose rows (vertices x 1 species) are the sampled rows."""
    return _predict_inputs(dict(verts=case["rows"], species=1), seed)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prep_setup(case, seed):
    _, xyz, cells = _mesh_inputs(case, seed)
    return dict(run=_run_setup, mesh=_tetmesh(xyz, cells),
                De=torch.exp(0.3 * _normal(cells.shape[0], _gen(seed, 1))))


def _run_setup(s):
    from dissolve_tp import assembler as A
    A.LUMP_MASS = 1
    asm = A.GPUSparseAssembler(s["mesh"])
    asm.assemble(s["De"], 50.0)
    return asm.d_indptr, asm.d_indices, asm.d_data


def _prep_assemble(case, seed):
    from dissolve_tp.assembler import GPUSparseAssembler
    xyz, cells, De, alpha, bc = _assemble_inputs(case, seed)
    return dict(run=_run_assemble, asm=GPUSparseAssembler(_tetmesh(xyz, cells)), De=De,
                alpha=alpha, bc=bc, lumped=int(case["lumped"]))


def _run_assemble(s):
    from dissolve_tp import assembler as A
    A.LUMP_MASS = s["lumped"]
    s["asm"].assemble(s["De"], 50.0, alpha=s["alpha"], bc_dofs=s["bc"])
    return s["asm"].d_data


def _prep_rhs(case, seed):
    from dissolve_tp.assembler import GPUSparseAssembler
    xyz, cells, u, f, bc = _rhs_inputs(case, seed)
    return dict(run=_run_rhs, asm=GPUSparseAssembler(_tetmesh(xyz, cells)), u=u, f=f, bc=bc,
                lumped=int(case["lumped"]))


def _run_rhs(s):
    from dissolve_tp import assembler as A
    A.LUMP_MASS = s["lumped"]
    return s["asm"].assemble_rhs(s["u"], 50.0, f=s["f"], bc_dofs=s["bc"], bc_value=0.25)


def _prep_apply(case, seed):
    import ceed_operators as C
    g, xyz, cells = _mesh_inputs(case, seed)
    V = xyz.shape[0]
    mesh_data = C.extract_ceed_mesh_data(_tetmesh(xyz, cells))
    De, u = torch.exp(0.3 * _normal(V, g)), _rand(V, g)
    op = C.CeedDiffusionMassOp(C.make_ceed(True)[0], mesh_data, De, 50.0)
    return dict(run=_run_apply, op=op, u=u, out=torch.empty_like(u))


def _run_apply(s):
    return s["op"].apply(s["u"], s["out"])


def _prep_transport(case, seed):
    import solvers
    from dissolve_tp.assembler import GPUSparseAssembler
    xyz, cells, De, alpha, u, bc = _transport_inputs(case, seed)
    mesh = _tetmesh(xyz, cells)
    field = lambda a: types.SimpleNamespace(  # noqa: E731
        x=types.SimpleNamespace(array=a), function_space=types.SimpleNamespace(mesh=mesh))
    de = field(De.cpu().numpy())
    de._solver_inv_dt, de._solver_bc_dofs = 20.0, bc.cpu().numpy()
    s = dict(run=_run_transport, de=de, alpha=alpha.cpu().numpy(), u_old=u.cpu().numpy(),
             rtol=case["rtol"], u=field(u.cpu().numpy().copy()),
             name="u %s %d" % (sorted(case.items()), seed))
    # the time loop's earlier steps have registered the geometry and cached the solver
    solvers.set_shared_geometry(GPUSparseAssembler(mesh))
    _run_transport(s)
    return s


def _run_transport(s):
    import solvers
    from dissolve_tp import assembler as A
    A.LUMP_MASS = 1
    s["u"].x.array[:] = s["u_old"]
    solvers.solve_transport(s["name"], None, None, s["u"], rtol=s["rtol"], max_it=5000,
                            use_gpu=True, de_field=s["de"], alpha_field=s["alpha"],
                            u_old=s["u_old"], bc_value=1.0)
    return s["u"].x.array


def _prep_plain(case, seed):
    from dissolve_tp.transport import PlainTransport
    xyz, cells, coef, u0, _ = _step_inputs(case, seed)
    D, k = _species(case["species"])
    tr = PlainTransport(_tetmesh(xyz, cells), coef, D, k, 0.02, rtol=case["rtol"])
    return dict(run=_run_plain, tr=tr, u=[u0[:, s].contiguous() for s in range(tr.S)])


def _run_plain(s):
    for a, b in zip(s["tr"].U, s["u"]):
        a.copy_(b)
    s["tr"].step(sync=False)
    return s["tr"].U


def _prep_step(case, seed):
    from dissolve_tp.transport import BatchedTransport
    xyz, cells, coef, u0, u1 = _step_inputs(case, seed)
    D, k = _species(case["species"])
    tr = BatchedTransport(_tetmesh(xyz, cells), coef, D, k, 0.02, rtol=case["rtol"],
                          inner_fp32=case["fp32"], guess=case["guess"], delta=0.01)
    s = dict(run=_run_step, tr=tr, u0=u0, u1=u1)
    if case["host"]:
        s.update(run=_run_step_host, u=u1.cpu().pin_memory(), out=torch.empty_like(
            u1, device="cpu").pin_memory())
    return s


def _run_step(s):
    # one step from two known time levels (a restart), so that every pass does the same work
    s["tr"].set_state(s["u1"], s["u0"])
    s["tr"].step(sync=False)
    return s["tr"].U


def _run_step_host(s):
    s["tr"].set_state(s["u1"], s["u0"])
    s["tr"].step_host(s["u"], s["out"])
    return s["out"]


def _prep_gyroid(case, seed):
    from dissolve_tp.coupled import GyroidStep
    xyz, cells, phi, coef, u0 = _gyroid_inputs(case, seed)
    g = GyroidStep(_tetmesh(xyz, cells), phi, coef, rtol=case["rtol"],
                   h=2.0 * math.pi / case["nx"])
    return dict(run=_run_gyroid, g=g, phi=phi, u=u0)


def _run_gyroid(s):
    s["g"].phi.copy_(s["phi"])
    s["g"].set_state(s["u"])
    s["g"].step(sync=False)
    return s["g"].tr.U, s["g"].phi


def _prep_batch(case, seed):
    from dissolve_tp.batch import MeshBatch
    boxes, D, k, u = _batch_inputs(case, seed)
    return dict(run=_run_batch, u=u, b=MeshBatch([_tetmesh(*b) for b in boxes], D, k, 0.02,
                                                 rtol=case["rtol"]))


def _run_batch(s):
    s["b"].set_state(s["u"])
    s["b"].step(sync=False)
    return s["b"].U


def _prep_predict(case, seed):
    up, un, nx, phi, ng, ops = _predict_inputs(case, seed)
    D, k = _species(case["species"])
    mlp = _mlp(seed)
    mlp.fit_normalization([(up, un, nx)], case["species"], D, k, phi, ng, ops=[ops])
    return dict(run=_run_predict, mlp=mlp, up=up, un=un, phi=phi, ng=ng, ops=ops, D=D, k=k,
                S=case["species"])


def _run_predict(s):
    return s["mlp"].predict(s["un"], s["up"], s["S"], s["un"].shape[1], s["D"], s["k"], s["phi"],
                            s["ng"], ops=s["ops"])


def _prep_gradient(case, seed):
    up, un, nx, phi, ng, ops = _gradient_fields(case, seed)
    mlp = _mlp(seed)
    mlp.fit_normalization([(up, un, nx)], 1, [1.0], [0.5], phi, ng, ops=[ops])
    mlp.add_pairs([(up, un, nx)], 1, 1, [1.0], [0.5], phi, ng, ops=[ops])
    return dict(run=_run_gradient, mlp=mlp, rows=case["rows"])


def _run_gradient(s):
    return s["mlp"].gradient(0, s["rows"])


_PREPARE = dict(setup=_prep_setup, assemble=_prep_assemble, rhs=_prep_rhs, apply=_prep_apply,
                transport=_prep_transport, plain=_prep_plain, step=_prep_step,
                gyroid=_prep_gyroid, batch=_prep_batch, predict=_prep_predict,
                gradient=_prep_gradient)


# ------------------------------------------------------------------ work
def _counts(nx, ny, nz):
    """cells, vertices and CSR entries (V + 2 E) of a Kuhn-split box."""
    V = (nx + 1) * (ny + 1) * (nz + 1)
    E = (nx * (ny + 1) * (nz + 1) + ny * (nx + 1) * (nz + 1) + nz * (nx + 1) * (ny + 1) +
         nx * ny * (nz + 1) + ny * nz * (nx + 1) + nx * nz * (ny + 1) + nx * ny * nz)
    return 6 * nx * ny * nz, V, V + 2 * E


def work(case):
    """Bytes: the mesh (16 per cell, 24 per vertex), the coefficients and fields read once, the
    results written once.  Flops: the element arithmetic (about 100 per cell), and for a solve
    the products of about four iterations per cell of the longest side."""
    k = case["kind"]
    if k == "predict":
        V, S = case["verts"], case["species"]
        return dict(bytes=V * (16.0 + S * (4 * 8 + 4)), flops=2.0 * V * S * (16 * 64 + 64 * 64 + 64))
    if k == "gradient":
        return dict(bytes=case["rows"] * 36.0 + 4 * 5313 * 2,
                    flops=6.0 * case["rows"] * (16 * 64 + 64 * 64 + 64))
    if k == "batch":
        sizes = np.random.default_rng(17 + case["meshes"]).integers(
            case["n_min"], case["n_max"] + 1, case["meshes"])
        c = [_counts(n, n, n) for n in sizes]
        return dict(bytes=float(sum(16 * a + 40 * b for a, b, _ in c)),
                    flops=float(sum(100 * a + 2 * z * 4 * n for (a, _, z), n in zip(c, sizes))))
    n, V, nnz = _counts(case["nx"], case["ny"], case["nz"])
    side = max(case["nx"], case["ny"], case["nz"])
    mesh = 16.0 * n + 24.0 * V
    if k == "setup":
        return dict(bytes=mesh + 8 * n + 4 * V + 12 * nnz, flops=100.0 * n)
    if k == "assemble":
        coef = 8 * (V if case["vertex_coef"] else n) * (2 if case["alpha"] else 1)
        return dict(bytes=mesh + coef + 8 * nnz, flops=100.0 * n)
    if k == "rhs":
        return dict(bytes=mesh + 8 * V * (3 if case["source"] else 2), flops=60.0 * n)
    if k == "apply":
        return dict(bytes=mesh + 8 * n + 16 * V, flops=120.0 * n)
    S = {"transport": 1, "gyroid": 3}.get(k) or case["species"]
    return dict(bytes=mesh + 8 * n + 16 * V * S, flops=100.0 * n + 2.0 * nnz * S * 4 * side)


# ------------------------------------------------------------------ exact results (64 bits)
def _element(xyz, cells):
    """Per cell: |det J| (n) and K / De = |det J| / 6 grad_i . grad_j (n, 4, 4)."""
    x = xyz[cells.long()]
    J = (x[:, 1:] - x[:, :1]).transpose(1, 2)  # columns are the edges
    e = [J[:, :, a] for a in range(3)]
    adj = torch.stack([torch.linalg.cross(e[1], e[2]), torch.linalg.cross(e[2], e[0]),
                       torch.linalg.cross(e[0], e[1])], 1)
    det = (e[0] * adj[:, 0]).sum(1)
    gr = adj / det[:, None, None]
    gr = torch.cat([-gr.sum(1, keepdim=True), gr], 1)
    dJ = det.abs()
    return dJ, dJ[:, None, None] / 6.0 * (gr @ gr.transpose(1, 2))


def _csr(xyz, cells, blocks):
    """Sparse CSR tensor of the (n, 4, 4) element blocks (sorted columns)."""
    V, c = xyz.shape[0], cells.long()
    r = c[:, :, None].expand(-1, 4, 4).reshape(-1)
    q = c[:, None, :].expand(-1, 4, 4).reshape(-1)
    return torch.sparse_coo_tensor(torch.stack([r, q]), blocks.reshape(-1),
                                   (V, V)).coalesce().to_sparse_csr()


def _mass(dJ, lumped):
    eye = torch.eye(4, dtype=torch.float64, device=dJ.device)
    M = 5.0 * eye if lumped else eye + 1.0
    return dJ[:, None, None] / 120.0 * M


def _cell(v, cells):
    return v if v.shape[0] == cells.shape[0] else v[cells.long()].mean(1)


def _operator(xyz, cells, De, alpha, inv_dt, lumped=True):
    dJ, K = _element(xyz, cells)
    a = inv_dt + (0.0 if alpha is None else _cell(alpha, cells))
    a = a * torch.ones_like(dJ)
    return _csr(xyz, cells, _cell(De, cells)[:, None, None] * K +
                a[:, None, None] * _mass(dJ, lumped)), dJ


def _dirichlet(A, bc):
    """Identity rows where bc (columns kept, as the operator's values are)."""
    n = A.shape[0]
    mask = torch.zeros(n, dtype=torch.bool, device="cuda")
    mask[bc.long()] = True
    crow, col, val = A.crow_indices(), A.col_indices(), A.values().clone()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), crow[1:] - crow[:-1])
    val = torch.where(mask[row], (row == col).double(), val)
    return torch.sparse_csr_tensor(crow, col, val, A.shape), mask


def _rhs(xyz, cells, dJ, u, f, inv_dt, lumped):
    w = inv_dt * u + (0.0 if f is None else f)
    wc = w[cells.long()]
    t = 5.0 * wc if lumped else wc + wc.sum(1, keepdim=True)
    return torch.zeros_like(u).index_add_(0, cells.long().reshape(-1),
                                          (dJ[:, None] / 120.0 * t).reshape(-1))


def _pcg(A, b, x, mask=None, tol=1e-15, most=6000):
    """Jacobi-PCG in 64 bits on the free rows, until the residual stops falling."""
    if mask is not None:
        x = torch.where(mask, b, x)
    n = A.shape[0]
    crow, col = A.crow_indices(), A.col_indices()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), crow[1:] - crow[:-1])
    d = torch.zeros_like(b)
    d[row[row == col]] = A.values()[row == col]
    dinv = 1.0 / d
    if mask is not None:
        dinv = torch.where(mask, torch.zeros_like(d), dinv)
    mv = lambda v: (A @ v[:, None])[:, 0]  # noqa: E731
    for _ in range(3):  # restarted from the true residual
        r = b - mv(x)
        if mask is not None:
            r[mask] = 0.0
        z = dinv * r
        p, rz, best = z.clone(), r @ z, float(torch.linalg.norm(b))
        for it in range(most):
            q = mv(p)
            if mask is not None:
                q[mask] = 0.0
            a = rz / (p @ q)
            x, r = x + a * p, r - a * q
            z = dinv * r
            new = r @ z
            p, rz = z + (new / rz) * p, new
            if it % 20 == 19 and not float(torch.linalg.norm(r)) > tol * best:
                break
    return x


def _solve(xyz, cells, De, alpha, inv_dt, u, f=None, bc=None, bc_value=0.0):
    A, dJ = _operator(xyz, cells, De, alpha, inv_dt)
    b = _rhs(xyz, cells, dJ, u, f, inv_dt, True)
    mask = None
    if bc is not None:
        A, mask = _dirichlet(A, bc)
        b = torch.where(mask, torch.full_like(b, bc_value), b)
    return _pcg(A, b, u.clone(), mask)


def _pad(cols):
    S = len(cols)
    out = torch.zeros((cols[0].shape[0], {1: 1, 2: 2, 3: 4, 4: 4}[S]), dtype=torch.float64,
                      device="cuda")
    out[:, :S] = torch.stack(cols, 1)
    return out


def _forward(p, X):
    W1, b1 = p[:1024].reshape(64, 16), p[1024:1088]
    W2, b2, w3, b3 = p[1088:5184].reshape(64, 64), p[5184:5248], p[5248:5312], p[5312]
    h = torch.relu(X @ W1.T + b1)
    return torch.relu(h @ W2.T + b2) @ w3 + b3


def _features(up, un, nx, phi, ng, ops, S, D, k):
    """The network's normalised inputs in 64 bits, rows = vertex * S + species."""
    V = un.shape[0]
    cut = lambda t: t[:, :S].reshape(-1)  # noqa: E731
    rep = lambda t: t[:, None].expand(V, S).reshape(-1)  # noqa: E731
    logD = torch.log(torch.tensor(D, dtype=torch.float64, device="cuda"))
    kk = torch.tensor(k, dtype=torch.float64, device="cuda")
    cols = [(rep(phi), phi), (rep(ng), ng), (cut(un), cut(un)), (cut(up), cut(up)),
            (cut(un - up), cut(un - up)), (logD.repeat(V), logD), (kk.repeat(V), kk), None,
            (cut(ops[0]), cut(ops[0])), (cut(ops[1]), cut(ops[1]))]
    X = torch.zeros((V * S, 16), dtype=torch.float64, device="cuda")
    for f, c in enumerate(cols):
        if c is None:
            X[:, f] = 1.0
        else:
            sd = c[1].std(correction=0)
            X[:, f] = (c[0] - c[1].mean()) * (1.0 / sd if float(sd) > 1e-12 else 1.0)
    T = cut(nx - un)
    return X, T / T.std(correction=0)


def exact(case, seed):
    k = case["kind"]
    if k == "setup":
        _, xyz, cells = _mesh_inputs(case, seed)
        De = torch.exp(0.3 * _normal(cells.shape[0], _gen(seed, 1)))
        return None, None, _operator(xyz, cells, De, None, 50.0)[0].values()
    if k == "assemble":
        xyz, cells, De, alpha, bc = _assemble_inputs(case, seed)
        A = _operator(xyz, cells, De, alpha, 50.0, case["lumped"])[0]
        return (A if bc is None else _dirichlet(A, bc)[0]).values()
    if k == "rhs":
        xyz, cells, u, f, bc = _rhs_inputs(case, seed)
        b = _rhs(xyz, cells, _element(xyz, cells)[0], u, f, 50.0, case["lumped"])
        if bc is not None:
            b[bc.long()] = 0.25
        return b
    if k == "apply":
        g, xyz, cells = _mesh_inputs(case, seed)
        De, u = torch.exp(0.3 * _normal(xyz.shape[0], g)), _rand(xyz.shape[0], g)
        return (_operator(xyz, cells, De, None, 50.0, False)[0] @ u[:, None])[:, 0]
    if k == "transport":
        xyz, cells, De, alpha, u, bc = _transport_inputs(case, seed)
        return _solve(xyz, cells, De, alpha, 20.0, u, bc=bc, bc_value=1.0).cpu().numpy()
    if k in ("plain", "step"):
        xyz, cells, coef, u0, u1 = _step_inputs(case, seed)
        D, kk = _species(case["species"])
        u = u0 if k == "plain" else u1
        one = torch.ones(cells.shape[0], dtype=torch.float64, device="cuda")
        x = [_solve(xyz, cells, D[s] * coef, kk[s] * one, 50.0, u[:, s].contiguous())
             for s in range(case["species"])]
        if k == "plain":
            return x
        return torch.stack(x, 1).cpu() if case["host"] else _pad(x)
    if k == "gyroid":
        xyz, cells, phi, coef, u = _gyroid_inputs(case, seed)
        eps = 1.5 * 2.0 * math.pi / case["nx"]
        H = 0.5 * (1.0 + phi / eps + torch.sin(math.pi * phi / eps) / math.pi)
        H = torch.where(phi > eps, torch.ones_like(H),
                        torch.where(phi < -eps, torch.zeros_like(H), H))
        hv = 2.0 * H
        one = torch.ones(cells.shape[0], dtype=torch.float64, device="cuda")
        x = [_solve(xyz, cells, D_S[s] * coef, K_S[s] * one + (_cell(hv, cells) if s == 0 else 0.0),
                    50.0, u[:, s].contiguous(), f=2.0 * hv * u[:, 0] if s == 2 else None)
             for s in range(3)]
        return _pad(x), phi - 0.02 * 0.01 * (1.0 + 0.5 * x[1])
    if k == "batch":
        boxes, D, kk, u = _batch_inputs(case, seed)
        out, at = [], 0
        for (xyz, cells), d, q in zip(boxes, D, kk):
            one = torch.ones(cells.shape[0], dtype=torch.float64, device="cuda")
            out.append(_solve(xyz, cells, d * one, q * one, 50.0, u[at:at + xyz.shape[0]]))
            at += xyz.shape[0]
        return torch.cat(out)
    if k == "predict":
        up, un, nx, phi, ng, ops = _predict_inputs(case, seed)
        D, kk = _species(case["species"])
        X, _ = _features(up, un, nx, phi, ng, ops, case["species"], D, kk)
        return _forward(_mlp_params(seed).double(), X)
    up, un, nx, phi, ng, ops = _gradient_fields(case, seed)
    X, T = _features(up, un, nx, phi, ng, ops, 1, [1.0], [0.5])
    p = _mlp_params(seed).double().requires_grad_(True)
    e = _forward(p, X) - T
    (e * e).mean().backward()
    return p.grad, (e * e).sum().reshape(1)

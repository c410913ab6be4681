"""The cluster engine (one thread-block cluster per system) and the exchange engine (the
same passes on every SM) against the grid and graph engines: every element type and column
count, Dirichlet rows, systems whose row ranges leave CTAs empty or partly filled, both
sides of the size where one engine hands over to the other, and many systems at once.

Bars: each solve converges on its FP64 residual (||b - A x|| <= rtol ||b||); solutions of
two engines at rtol 1e-11 agree within 1e-8 relative L2 (the residual rule times the
condition number of the Jacobi-scaled operator, below 1e3 on these meshes), every lane's
reported residual is the residual of the returned x within 1 %."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(shape, S, fp32, bc, seed=0):
    import torch
    from dissolve_tp.assembler import GPUSparseAssembler
    from dissolve_tp.krylov import CsrOperator
    from dissolve_tp.mesh import face_dofs, kuhn_cube
    m = kuhn_cube(shape, 0.2, seed=seed)
    rng = np.random.default_rng(seed + 1)
    asm = GPUSparseAssembler(m)
    dofs = face_dofs(m, 0, "min") if bc else None
    coef = np.exp(0.3 * rng.standard_normal(m.n_cells))
    asm.assemble(coef, 0.0)  # stiffness alone; the diagonal carries the mass
    ld = {1: 1, 2: 2, 3: 4, 4: 4}[S]
    V = m.n_verts
    diag = torch.zeros((V, ld), dtype=torch.float64, device="cuda")
    diag[:, :S] = torch.from_numpy(rng.uniform(0.5, 1.0, (V, S)) * 50.0 / V)
    mask = asm._dm.bc_mask(dofs) if bc else None
    K32 = asm.d_data.float() if fp32 else None
    op = CsrOperator(asm.d_indptr, asm.d_indices, asm.d_data.clone(), K32=K32, diag64=diag,
                     diag32=diag.float() if fp32 else None, bc_mask=mask,
                     dscale=[1.0, 0.7, 2.6, 1.3][:S], S=S, ld=ld)
    b = torch.zeros((V, ld), dtype=torch.float64, device="cuda")
    b[:, :S] = torch.from_numpy(rng.uniform(-1.0, 1.0, (V, S)) / V)
    return asm, op, b


def _check(op, sol, res, b, rtol):
    import torch
    S = op.S
    assert res["converged"], res
    r = (b - op.apply(sol.x))[:, :S]
    rn = torch.linalg.norm(r, dim=0).cpu().numpy()
    assert np.all(res["rnorm"] <= rtol * res["bnorm"])
    assert np.all(np.abs(rn - res["rnorm"]) <= 0.01 * res["rnorm"] + 1e-14 * res["bnorm"])


@pytest.mark.parametrize("n,S,fp32,bc,engine", [
    (1, 1, False, False, "cluster"), (3, 1, True, False, "cluster"),
    (7, 2, False, True, "cluster"), (9, 3, True, True, "cluster"),
    (12, 4, True, False, "cluster"), (10, 4, False, False, "cluster"),
    (16, 1, False, True, "cluster"), (20, 2, True, False, "cluster"),
    (23, 3, True, False, "cluster"), (28, 1, False, False, "cluster"),
    (33, 1, True, False, "cluster"), (29, 1, False, True, "exchange"),
    (35, 1, True, True, "exchange"), (26, 3, True, True, "exchange"),
    (27, 4, True, False, "exchange"), (28, 2, False, False, "exchange"),
    (24, 3, False, False, "exchange"), (22, 4, False, True, "exchange"),
    (34, 2, True, False, "exchange"), (48, 1, False, False, "exchange"),
    (44, 3, True, False, "exchange"), (55, 3, True, True, "exchange"),
    (56, 3, True, False, "exchange"), (54, 4, True, True, "exchange")])
def test_engine_matches_grid_engine(cuda_device, monkeypatch, n, S, fp32, bc, engine):
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(n, S, fp32, bc)
    kw = dict(rtol=1e-11, max_it=4000, inner_fp32=fp32, delta=0.01)
    one = PersistentCG(op, **kw)
    monkeypatch.setenv("DISSOLVE_PCG_PIPE", "0")
    grid = PersistentCG(op, **kw)
    assert one.engine()[engine], one.engine()
    assert not grid.engine()["cluster"] and not grid.engine()["exchange"]
    out = []
    for sol in (one, grid):
        sol.b.copy_(b)
        sol.x.zero_()
        res = sol.solve()
        _check(op, sol, res, b, 1e-11)
        out.append(sol.x.clone())
    assert torch.linalg.norm(out[0] - out[1]) <= 1e-8 * torch.linalg.norm(out[1])
    # bit-reproducible
    one.x.zero_()
    one.solve()
    assert torch.equal(one.x, out[0])


@pytest.mark.parametrize("fp32", [True, False])
def test_cluster_queue_of_systems_matches_graph_engine(cuda_device, fp32):
    """more systems than clusters, of very different sizes; FP32 and FP64"""
    import torch
    from dissolve_tp.batch import MeshBatch, uneven_batch_inputs
    meshes, D, k = uneven_batch_inputs(40, 1, 14, seed=3)
    mb = MeshBatch(meshes, D, k, 0.02, rtol=1e-11, inner_fp32=fp32)
    assert mb.solver.cluster()
    ref = MeshBatch(meshes, D, k, 0.02, rtol=1e-11, inner_fp32=fp32,
                    cg=dict(group=2, block=128, rows_per_tile=128, use_graph_loop=False))
    assert not ref.solver.cluster()
    u = np.random.default_rng(5).uniform(0, 1, int(mb.vert_ptr[-1]))
    for x in (mb, ref):
        x.set_state(u)
        r = x.step()
        assert r["converged"] and np.all(r["rnorm"] <= 1e-11 * r["bnorm"])
    assert torch.linalg.norm(mb.U - ref.U) <= 1e-9 * torch.linalg.norm(ref.U)


def test_cluster_failures_are_reported_per_lane(cuda_device):
    """max_it, a non-SPD column and a NaN column end with their own status; the healthy
    column of the same solve converges."""
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(8, 3, False, False)
    sol = PersistentCG(op, rtol=1e-10, max_it=3)
    sol.b.copy_(b)
    res = sol.solve()
    assert sol.engine()["cluster"] and res["status"] == 6 and res["iterations"] == 3
    op.set_scales(dscale=[1.0, -1.0, 1.0])
    sol = PersistentCG(op, rtol=1e-10, max_it=500)
    sol.b.copy_(b)
    sol.b[3, 2] = float("nan")
    res = sol.solve()
    assert list(res["lane_status"]) == [0, 7, 8], res
    sol.b[:, 1:].zero_()
    sol.x.zero_()
    res = sol.solve()  # zero right-hand sides: converged at once
    assert list(res["lane_status"]) == [0, 0, 0] and list(res["lane_iterations"][1:]) == [0, 0]
    assert torch.all(sol.x[:, 1:] == 0)


def test_cluster_solve_is_captured_in_a_graph(cuda_device):
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(11, 3, True, True)
    sol = PersistentCG(op, rtol=1e-10, max_it=2000, inner_fp32=True)
    sol.b.copy_(b)
    sol.x.zero_()
    ref = sol.solve()
    x = sol.x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sol.run()
    for _ in range(2):
        sol.x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(sol.x, x) and sol.result()["iterations"] == ref["iterations"]


@pytest.mark.parametrize("n,S,fp32", [(30, 1, False), (26, 3, True)])
def test_exchange_wait_runs_out_then_recovers(cuda_device, n, S, fp32):
    """Every wait expects a pass number that never comes: the solve ends with TP_ERR_TIMEOUT
    after the 1 ms limit and the handle then solves with the same bits as before."""
    import time

    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(n, S, fp32, False)
    sol = PersistentCG(op, rtol=1e-10, max_it=4000, inner_fp32=fp32)
    assert sol.engine()["exchange"]
    sol.b.copy_(b)
    ref = sol.solve()
    x = sol.x.clone()
    assert ref["converged"]
    sol.set_wait_limit(1e-3, missing_arrivals=1)
    sol.x.zero_()
    t0 = time.perf_counter()
    res = sol.solve()
    assert res["status"] == 9 and list(res["lane_status"]) == [9] * S
    assert time.perf_counter() - t0 < 1.0
    sol.set_wait_limit(0.0, 0)
    sol.x.zero_()
    res = sol.solve()
    assert res["converged"] and res["iterations"] == ref["iterations"]
    assert torch.equal(sol.x, x)


def test_exchange_solve_is_captured_in_a_graph(cuda_device):
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(28, 3, True, True)
    sol = PersistentCG(op, rtol=1e-10, max_it=2000, inner_fp32=True)
    assert sol.engine()["exchange"]
    sol.b.copy_(b)
    ref = sol.solve()
    x = sol.x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sol.run()
    for _ in range(2):
        sol.x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(sol.x, x) and sol.result()["iterations"] == ref["iterations"]


@pytest.mark.parametrize("n,S,fp32", [(55, 3, True), (54, 4, True), (40, 1, False)])
def test_exchange_engine_with_long_rows(cuda_device, monkeypatch, n, S, fp32):
    """27-point rows: more entries than tensor memory holds per row, so the values are read
    from shared memory or L2."""
    import scipy.sparse as sp
    import torch
    from dissolve_tp.krylov import CsrOperator, PersistentCG
    t = sp.diags([np.ones(n - 1), np.ones(n), np.ones(n - 1)], [-1, 0, 1])
    A = (27.5 * sp.identity(n ** 3) - sp.kron(sp.kron(t, t), t)).tocsr()
    A.sort_indices()
    ld = {1: 1, 3: 4, 4: 4}[S]
    V = n ** 3
    K = torch.from_numpy(A.data).cuda()
    rng = np.random.default_rng(n)
    diag = torch.zeros((V, ld), dtype=torch.float64, device="cuda")
    diag[:, :S] = torch.from_numpy(rng.uniform(0.5, 1.0, (V, S)))
    op = CsrOperator(torch.from_numpy(A.indptr.astype(np.int32)).cuda(),
                     torch.from_numpy(A.indices.astype(np.int32)).cuda(), K,
                     K32=K.float() if fp32 else None, diag64=diag,
                     diag32=diag.float() if fp32 else None, dscale=[1.0, 0.7, 2.6, 1.3][:S], S=S,
                     ld=ld)
    b = torch.zeros((V, ld), dtype=torch.float64, device="cuda")
    b[:, :S] = torch.from_numpy(rng.uniform(-1.0, 1.0, (V, S)))
    kw = dict(rtol=1e-11, max_it=4000, inner_fp32=fp32, delta=0.01)
    one = PersistentCG(op, **kw)
    monkeypatch.setenv("DISSOLVE_PCG_PIPE", "0")
    grid = PersistentCG(op, **kw)
    assert one.engine()["exchange"] and not grid.engine()["exchange"]
    out = []
    for sol in (one, grid):
        sol.b.copy_(b)
        sol.x.zero_()
        _check(op, sol, sol.solve(), b, 1e-11)
        out.append(sol.x.clone())
    assert torch.linalg.norm(out[0] - out[1]) <= 1e-8 * torch.linalg.norm(out[1])

"""The engines that the cluster and exchange engines stand in front of, each asked for by name
and checked to be the one that runs: the conditional-node graph engine (tp_cg_* with
use_graph_loop = 2), and the streaming, window, tensor-memory and pipelined grid engines.

Bars: solutions at rtol 1e-10 agree with the oracle's direct solution within 1e-9 (FP64) or
1e-8 (FP32 inner) relative L2, as in the tests of the persistent engine."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_gpu_cluster import _operator
from test_gpu_solvers import _config1, _np

pytestmark = pytest.mark.gpu

GRID_ENGINES = {  # environment, engine() flags (window, tmem, pipelined)
    "stream": (dict(DISSOLVE_PCG_ENGINE="stream"), (False, False, False)),
    "cgw": (dict(DISSOLVE_PCG_CGT="0"), (True, False, False)),
    "cgt": (dict(DISSOLVE_PCG_PIPE="0"), (True, True, False)),
    "pipe": (dict(DISSOLVE_PCG_PIPE="1"), (True, True, True))}


def _grid_solver(monkeypatch, engine, op, **kw):
    from dissolve_tp.krylov import PersistentCG
    env, want = GRID_ENGINES[engine]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    sol = PersistentCG(op, inner_fp32=True, **kw)
    e = sol.engine()
    assert (e["window"], e["tmem"], e["pipelined"]) == want, e
    assert not e["cluster"] and not e["exchange"]
    return sol


@pytest.mark.parametrize("inner_fp32", [False, True])
def test_graph_engine_config1(cuda_device, inner_fp32):
    import torch
    from dissolve_tp import assembler as A, krylov as K
    m, bc, u0, asm, b = _config1(A)
    op = K.CsrOperator(asm.d_indptr, asm.d_indices, asm.d_data,
                       K32=asm.d_data.float() if inner_fp32 else None,
                       bc_mask=asm._dm.bc_mask(bc))
    ip, ix, A_ = asm.mat.getValuesCSR()
    xd = orc.direct_solve(ip, ix, A_, _np(b))
    its = {}
    for engine in ("graph", "auto"):
        sol = K.CGSolver(op, rtol=1e-10, max_it=3000, inner_fp32=inner_fp32, engine=engine)
        assert sol.cluster() == (engine == "auto")
        sol.b[:, 0].copy_(b)
        sol.x[:, 0].copy_(torch.from_numpy(u0))
        res = sol.solve()
        assert res["converged"] and res["rnorm"][0] <= 1e-10 * res["bnorm"][0], res
        x = _np(sol.x[:, 0])
        assert np.linalg.norm(x - xd) / np.linalg.norm(xd) < (1e-8 if inner_fp32 else 1e-9)
        assert np.all(x[bc] == 1.0)
        its[engine] = res["iterations"]
    if not inner_fp32:
        assert abs(its["graph"] - its["auto"]) <= 2, its


def test_graph_engine_reports_breakdown_and_max_it(cuda_device):
    from dissolve_tp import assembler as A, krylov as K
    m, bc, u0, asm, b = _config1(A)
    for vals, rtol, status in ((-asm.d_data, 1e-10, 7), (asm.d_data, 1e-14, 6)):
        op = K.CsrOperator(asm.d_indptr, asm.d_indices, vals)
        sol = K.CGSolver(op, rtol=rtol, max_it=5, engine="graph")
        assert not sol.cluster()
        sol.b[:, 0].copy_(b)
        res = sol.solve()
        assert not res["converged"] and res["status"] == status, res


def test_graph_engine_with_a_mass_matrix(cuda_device):
    """A mass matrix with diagonal entries only equals the same numbers given as a diagonal."""
    import torch
    from dissolve_tp import krylov as K
    asm, op, b = _operator(9, 2, False, True)
    ip = op.arrays["indptr"].long()
    rows = torch.repeat_interleave(torch.arange(op.n_rows, device="cuda"), ip[1:] - ip[:-1])
    M = (rows == op.arrays["indices"]).double() * 0.05
    kw = dict(bc_mask=op.arrays["bc_mask"], dscale=[1.0, 0.7], S=2)
    mass = K.CsrOperator(asm.d_indptr, asm.d_indices, op.arrays["K64"], M64=M,
                         cscale=[1.0, 2.0], **kw)
    diag = torch.full((op.n_rows, 2), 0.05, dtype=torch.float64, device="cuda")
    diag[:, 1] = 0.1
    ref = K.CsrOperator(asm.d_indptr, asm.d_indices, op.arrays["K64"], diag64=diag, **kw)
    x = []
    for o, cluster in ((mass, False), (ref, True)):
        sol = K.CGSolver(o, rtol=1e-11, max_it=2000)
        assert sol.cluster() == cluster
        sol.b.copy_(b)
        assert sol.solve()["converged"]
        x.append(sol.x.clone())
    assert torch.linalg.norm(x[0] - x[1]) <= 1e-9 * torch.linalg.norm(x[1])


def test_callers_choose_the_graph_engine(cuda_device):
    """BatchedTransport and PlainTransport with engine="graph", and MeshBatch with a launch
    shape, run the graph engine and agree with the default engines."""
    import torch
    from dissolve_tp import transport as T
    from dissolve_tp.batch import MeshBatch, uneven_batch_inputs
    from dissolve_tp.mesh import kuhn_cube
    m = kuhn_cube(9, 0.2, seed=0)
    rng = np.random.default_rng(1)
    coef = np.exp(0.3 * rng.standard_normal(m.n_cells))
    u0 = rng.uniform(0, 1, (m.n_verts, 2))
    for form in (T.BatchedTransport, T.PlainTransport):
        out = []
        for engine in ("graph", "persistent"):
            tr = form(m, coef, (1.0, 2.6), (0.5, 0.0), 0.02, rtol=1e-11, engine=engine)
            if engine == "graph":
                sols = tr.solvers if form is T.PlainTransport else [tr.solver]
                assert not any(s.cluster() for s in sols)
                if form is T.BatchedTransport:
                    assert tr.cg_config["engine"] == "graph" and "group" in tr.cg_config
            tr.set_state(u0)
            tr.step()
            out.append(tr.state())
        assert np.linalg.norm(out[0] - out[1]) <= 1e-9 * np.linalg.norm(out[1])
    meshes, D, k = uneven_batch_inputs(5, 4, 9, seed=1)
    us = []
    for cg in (None, dict(group=2, block=128, rows_per_tile=128), dict(engine="graph")):
        mb = MeshBatch(meshes, D, k, 0.02, rtol=1e-11, cg=cg)
        assert mb.solver.cluster() == (cg is None)
        assert mb.cg_config["engine"] == ("cluster" if cg is None else "graph")
        assert cg is None or mb.cg_config["group"] in (1, 2, 4, 8)
        mb.set_state(np.random.default_rng(5).uniform(0, 1, int(mb.vert_ptr[-1])))
        assert mb.step()["converged"]
        us.append(mb.U.clone())
    for u in us[1:]:
        assert torch.linalg.norm(u - us[0]) <= 1e-9 * torch.linalg.norm(us[0])


@pytest.mark.parametrize("n_big,fp32,cluster", [(30, False, True), (34, True, True),
                                                (42, True, False)])
def test_batch_of_two_cluster_sizes(cuda_device, n_big, fp32, cluster):
    """Nine meshes, one of them too large for the small clusters (solved on a stream of its
    own beside the others, also under capture) or for any cluster (the graph engine)."""
    import torch
    from dissolve_tp.batch import MeshBatch
    from dissolve_tp.mesh import kuhn_cube
    meshes = [kuhn_cube(n, 0.2, seed=n) for n in (5, 8, 3, n_big, 10, 7, 4, 9, 6)]
    D, k = np.linspace(0.5, 2.0, 9), np.linspace(0.0, 1.0, 9)
    kw = dict(rtol=1e-11, inner_fp32=fp32)
    mb = MeshBatch(meshes, D, k, 0.02, **kw)
    assert mb.solver.cluster() == cluster
    ref = MeshBatch(meshes, D, k, 0.02, cg=dict(group=2, block=128, rows_per_tile=128), **kw)
    u = np.random.default_rng(5).uniform(0, 1, int(mb.vert_ptr[-1]))
    for x in (mb, ref):
        x.set_state(u)
        r = x.step()
        assert r["converged"] and np.all(r["rnorm"] <= 1e-11 * r["bnorm"])
    assert torch.linalg.norm(mb.U - ref.U) <= 1e-9 * torch.linalg.norm(ref.U)
    if not cluster:
        return
    x0 = torch.from_numpy(u).cuda()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        mb.solver.run()
    for _ in range(2):
        mb.solver.x.view(-1).copy_(x0)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(mb.solver.x.view(-1), mb.U)


@pytest.mark.parametrize("engine", list(GRID_ENGINES))
def test_grid_engines_report_breakdown_and_max_it(cuda_device, monkeypatch, engine):
    asm, op, b = _operator(12, 2, True, False)
    sol = _grid_solver(monkeypatch, engine, op, rtol=1e-14, max_it=5)
    sol.b.copy_(b)
    res = sol.solve()
    assert res["status"] == 6 and res["iterations"] == 5, res
    op.set_scales(dscale=[1.0, -1.0])
    sol = _grid_solver(monkeypatch, engine, op, rtol=1e-10, max_it=500)
    sol.b.copy_(b)
    res = sol.solve()
    assert list(res["lane_status"]) == [0, 7] and res["status"] == 7, res


@pytest.mark.parametrize("engine", list(GRID_ENGINES))
def test_grid_engines_wait_runs_out_then_recovers(cuda_device, monkeypatch, engine):
    import torch
    asm, op, b = _operator(12, 2, True, False)
    sol = _grid_solver(monkeypatch, engine, op, rtol=1e-10, max_it=2000)
    sol.b.copy_(b)
    ref = sol.solve()
    assert ref["converged"], ref
    x = sol.x.clone()
    sol.set_wait_limit(1e-3, missing_arrivals=1)
    sol.x.zero_()
    assert list(sol.solve()["lane_status"]) == [9, 9]
    sol.set_wait_limit(0.0, 0)
    sol.x.zero_()
    res = sol.solve()
    assert res["converged"] and res["iterations"] == ref["iterations"]
    assert torch.equal(sol.x, x)

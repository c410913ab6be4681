"""Wait limits of the cluster and exchange engines that are shorter than the skew between
CTAs and warps: single waits run out at scattered places of a solve, while other CTAs go on.
Every such solve ends, either converged with the bits of an undisturbed solve or with
TP_ERR_TIMEOUT on every column, and the handle then solves as before."""
import pytest

from test_gpu_cluster import _operator

pytestmark = pytest.mark.gpu

LIMITS_NS = (1, 100, 300, 500, 700, 1000, 1500, 2000, 3000, 5000, 10000)


def _short_limits(op, b, engine, **kw):
    import torch
    from dissolve_tp.krylov import PersistentCG
    sol = PersistentCG(op, rtol=1e-10, max_it=2000, **kw)
    assert sol.engine()[engine], sol.engine()
    sol.b.copy_(b)
    ref = sol.solve()
    assert ref["converged"], ref
    x = sol.x.clone()
    for limit in LIMITS_NS * 3:
        sol.set_wait_limit(limit * 1e-9)
        sol.x.zero_()
        res = sol.solve()
        if res["status"] == 0:
            assert torch.equal(sol.x, x) and res["iterations"] == ref["iterations"]
        else:
            assert list(res["lane_status"]) == [9] * op.S, (limit, res)
    sol.set_wait_limit(0.0)
    sol.x.zero_()
    res = sol.solve()
    assert res["converged"] and res["iterations"] == ref["iterations"]
    assert torch.equal(sol.x, x)


@pytest.mark.parametrize("n,S,fp32", [(29, 1, False), (26, 3, True), (44, 3, True)])
def test_exchange_engine_with_short_wait_limits(cuda_device, n, S, fp32):
    asm, op, b = _operator(n, S, fp32, False)
    _short_limits(op, b, "exchange", inner_fp32=fp32)


@pytest.mark.parametrize("n,S,fp32", [(16, 1, False), (20, 3, True), (33, 1, True),
                                      (12, 4, False)])
def test_cluster_engine_with_short_wait_limits(cuda_device, n, S, fp32):
    """Among the places: a wait for the sums of a pass after which the others go on to an
    FP64 sweep (FP32 columns refresh often)."""
    asm, op, b = _operator(n, S, fp32, False)
    _short_limits(op, b, "cluster", inner_fp32=fp32)


def test_cluster_engine_meeting_runs_out_then_recovers(cuda_device):
    """Every wait expects something that never comes, the meeting before the first sweep
    among them."""
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(14, 3, True, True)
    sol = PersistentCG(op, rtol=1e-10, max_it=2000, inner_fp32=True)
    assert sol.engine()["cluster"]
    sol.b.copy_(b)
    ref = sol.solve()
    x = sol.x.clone()
    sol.set_wait_limit(1e-4, missing_arrivals=1)
    sol.x.zero_()
    assert list(sol.solve()["lane_status"]) == [9, 9, 9]
    sol.set_wait_limit(0.0, 0)
    sol.x.zero_()
    res = sol.solve()
    assert res["converged"] and res["iterations"] == ref["iterations"]
    assert torch.equal(sol.x, x)

"""A column of the cluster and exchange engines that stood still at the tolerance and is not
confirmed by the FP64 sweep: its search direction is gone, so it restarts along u = D^-1 r.

The column's tolerance is set a little below its FP64 residual after k iterations, where the
FP32 recurrence, which has drifted from that residual by a factor of 1e-7 to 1e-4, may lie
below.  max_it = m shows the same solve after m iterations.  The first iteration after the
sweep is then a step of steepest descent from the x of the one before; its residual is
computed here in FP64 (bar 1e-3: the step is taken in FP32, whose errors of a few 1e-7 come in
relative to a residual of the same size).  A step with the coefficients of the lost direction
about doubles the residual."""
import pytest

from test_gpu_cluster import _operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S,engine", [(10, 2, "cluster"), (13, 3, "cluster"),
                                        (26, 3, "exchange"), (55, 3, "exchange")])
def test_unconfirmed_column_restarts(cuda_device, n, S, engine):
    import torch
    from dissolve_tp.krylov import PersistentCG, SellPattern
    asm, op, b = _operator(n, S, True, False)
    sell = SellPattern(op.arrays["indptr"], op.arrays["indices"])
    ip = op.arrays["indptr"].long()
    rows = torch.repeat_interleave(torch.arange(op.n_rows, device="cuda"), ip[1:] - ip[:-1])
    kd = op.arrays["K64"][rows == op.arrays["indices"]]
    dinv = 1.0 / (op.dscale[0] * kd + op.arrays["diag64"][:, 0])

    def solve(m, rtol0):
        sol = PersistentCG(op, rtol=[rtol0] + [1e-13] * (S - 1), max_it=m, inner_fp32=True,
                           sell=sell)
        assert sol.engine()[engine]
        sol.b.copy_(b)
        return sol.solve()["rnorm"][0], sol

    def steepest_descent(x):
        r = b - op.apply(x)
        u = torch.zeros_like(r)
        u[:, 0] = dinv * r[:, 0]
        Au = op.apply(u)[:, 0]
        r, u = r[:, 0], u[:, 0]
        return float(torch.linalg.norm(r - torch.dot(r, u) / torch.dot(u, Au) * Au))

    bnorm = float(torch.linalg.norm(b[:, 0]))
    checked = 0
    for k in range(4, 40):
        rk, _ = solve(k, 1e-14)
        for t in (1e-7, 1e-6, 1e-5, 5e-5):
            rtol0 = rk * (1.0 - t) / bnorm
            if abs(solve(k + 1, rtol0)[0] / rk - 1.0) > 1e-9:
                continue  # still running at k: the recurrence is not below the tolerance
            prev = None
            for m in range(k + 1, k + 80):
                r, sol = solve(m, rtol0)
                if abs(r / rk - 1.0) > 1e-9:  # the first iteration after the sweep
                    want = steepest_descent(prev.x)
                    assert abs(r / want - 1.0) < 1e-3, (k, t, m, r / rk, want / rk)
                    checked += 1
                    break
                prev = sol
            break
        if checked == 2:
            break
    assert checked

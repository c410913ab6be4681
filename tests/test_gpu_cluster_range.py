"""Right-hand sides far from 1 in the cluster and exchange engines."""
import pytest

from test_gpu_cluster import _operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S,engine", [(12, 1, "cluster"), (10, 3, "cluster"),
                                        (30, 1, "exchange"), (24, 3, "exchange")])
@pytest.mark.parametrize("power", [-400, -330, 200, 330, 400])
def test_solution_scales_with_the_right_hand_side(cuda_device, n, S, engine, power):
    """A b scaled by a power of two scales every number of an FP64 solve by a power of two
    while the squared norms stay in range (2^+-800 here, after 1 / V and twenty decades of
    residual): the same iterations, and the same x scaled, bit for bit."""
    import torch
    from dissolve_tp.krylov import PersistentCG
    asm, op, b = _operator(n, S, False, False)
    sol = PersistentCG(op, rtol=1e-10, max_it=2000)
    assert sol.engine()[engine]
    sol.b.copy_(b)
    ref = sol.solve()
    x = sol.x.clone()
    assert ref["converged"]
    sol.b.copy_(b * 2.0 ** power)
    sol.x.zero_()
    res = sol.solve()
    assert res["converged"], res
    assert list(res["lane_iterations"]) == list(ref["lane_iterations"])
    assert torch.equal(sol.x, x * 2.0 ** power)

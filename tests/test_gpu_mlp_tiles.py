"""Warm-start network at the edges of its tiles: training gradients around one 64-row chunk
(16-row warp tiles).

Bars as for the other sizes of the same kernels: the oracle rounds to BF16 at the same points,
gradients within 5e-3 (norm-wise per parameter block)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo


def _params(seed):
    rng = np.random.default_rng(seed)
    p = mo.init_params(seed).astype(np.float64)
    p[mo.OFF_B1:mo.OFF_W2] = rng.normal(0, 0.2, mo.H)
    p[mo.OFF_B2:mo.OFF_W3] = rng.normal(0, 0.2, mo.H)
    p[mo.OFF_B3] = 0.1
    return p.astype(np.float32), rng


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 15, 17, 63, 65, 128, 19009])
def test_gradient_at_chunk_edges(cuda_device, rows):
    import torch

    from dissolve_tp.mlp import WarmStartMLP
    p, rng = _params(21)
    X = rng.normal(0, 1, (rows, mo.IN))
    X[:, 7] = 1.0
    X[:, mo.NFEAT:] = 0.0
    X = mo.bf16(X)
    T = rng.normal(0, 1, rows).astype(np.float32)
    m = WarmStartMLP(cuda_device, capacity_rows=rows)
    m.params.copy_(torch.from_numpy(p))
    m.X[:rows].copy_(torch.from_numpy(X.astype(np.float32)).to(torch.bfloat16))
    m.T[:rows].copy_(torch.from_numpy(T))
    m.rows = rows
    g, loss = m.gradient(0, rows)
    g = g.cpu().numpy().astype(np.float64)
    lo, go = mo.loss_and_grad(p, X, T.astype(np.float64))
    assert abs(float(loss.item()) - lo) <= 2e-3 * lo
    for a, b in ((mo.OFF_W1, mo.OFF_B1), (mo.OFF_B1, mo.OFF_W2), (mo.OFF_W2, mo.OFF_B2),
                 (mo.OFF_B2, mo.OFF_W3), (mo.OFF_W3, mo.OFF_B3), (mo.OFF_B3, mo.P)):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= 5e-3 * np.linalg.norm(go[a:b])

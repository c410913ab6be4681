"""Warm-start network at the edges of its tiles: training gradients around one 64-row chunk
(16-row warp tiles), inference around one 128-row half, one 256-row tile and one full grid.

Bars as for the other sizes of the same kernels: the oracle rounds to BF16 at the same points,
gradients within 5e-3 (norm-wise per parameter block), outputs within 2e-3 (max-norm)."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("species", [1, 2, 3, 4])
@pytest.mark.parametrize("rows", [1, 127, 129, 256, 257, 113700])
def test_inference_at_tile_edges(cuda_device, rows, species):
    """x_out and y of every row (within 2e-3 of the largest output of 1,000 such rows), and
    nothing outside them: the padding columns and the vertices past the last one keep their
    values."""
    import torch

    from dissolve_tp.mlp import WarmStartMLP
    p, rng = _params(22)
    V = -(-rows // species)
    n = max(V, 1000)
    ld = species + (species == 3)
    m = WarmStartMLP(cuda_device, base="extrapolate")
    m.params.copy_(torch.from_numpy(p))
    m.sigma = 0.01
    U = rng.uniform(0, 1, (n, species))
    Up = U + rng.normal(0, 0.05, (n, species))
    D, k = [1.0, 0.7, 2.6, 1.3][:species], [0.5, 0.0, 0.2, 0.1][:species]
    X = mo.features(U, Up, None, None, np.log(D), k, m.mean, m.istd)
    yo, _ = mo.forward(p, X)
    bar = 2e-3 * np.abs(yo).max()
    U, Up, yo = U[:V], Up[:V], yo[: V * species]
    Ud = torch.zeros((V, ld), dtype=torch.float64, device=cuda_device)
    Upd = torch.zeros_like(Ud)
    Ud[:, :species] = torch.from_numpy(U)
    Upd[:, :species] = torch.from_numpy(Up)
    y = m.predict(Ud, Upd, species, ld, D, k).cpu().numpy().astype(np.float64)
    assert np.abs(y - yo).max() <= bar
    x = torch.full((V + 1, ld), 7.0, dtype=torch.float64, device=cuda_device)
    m.predict(Ud, Upd, species, ld, D, k, x_out=x[:V])
    assert not m.timed_out()
    xo = 2.0 * U - Up + m.sigma * yo.reshape(V, species)
    got = x.cpu().numpy()
    assert np.abs(got[:V, :species] - xo).max() <= bar * m.sigma + 1e-12
    assert np.all(got[:V, species:] == 7.0) and np.all(got[V] == 7.0)

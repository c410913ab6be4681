"""The tile tables built on the GPU (tp_tiles_create): one partition of the rows into tiles
of nearby rows whatever the mesh, and assemblies equal to the row walk bit for bit, at the
sizes where the bisection and the table builder can go wrong: one cell, row counts around a
tile, tiles of 32 to 256 rows, flat and anisotropic boxes, coincident coordinates, vertices
that no cell uses, a vertex of high degree."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(nx, ny, nz, scale=(1.0, 1.0, 1.0)):
    from dissolve_tp.mesh import _KUHN_PERMS
    s = (1, nx + 1, (nx + 1) * (ny + 1))
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    xyz = np.stack([i.ravel() * scale[0], j.ravel() * scale[1], k.ravel() * scale[2]], 1)
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    base = (i + j * s[1] + k * s[2]).ravel()
    cells = []
    for p in _KUHN_PERMS:
        v = [base]
        for a in p:
            v.append(v[-1] + s[a])
        cells.append(np.stack(v, 1))
    return xyz.astype(np.float64), np.stack(cells, 1).reshape(-1, 4).astype(np.int32)


def _star(n):
    """n cells around one vertex: triangles of a fan on a sphere-like cap"""
    t = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(t), np.sin(t), np.zeros(n)], 1)
    xyz = np.concatenate([[[0.0, 0.0, 1.0], [0.0, 0.0, -0.5]], ring])
    q = np.arange(n)
    return xyz, np.stack([np.zeros(n, int), np.ones(n, int), 2 + q, 2 + (q + 1) % n],
                         1).astype(np.int32)


def _mesh(kind):
    if kind == "one_cell":
        return _box(1, 1, 1)[0][:8], np.array([[0, 1, 3, 7]], np.int32)  # 4 unused vertices
    if kind == "rows_63":
        return _box(2, 2, 6)
    if kind == "rows_64":
        return _box(3, 3, 3)
    if kind == "rows_65":
        x, c = _box(3, 3, 3)
        return np.concatenate([x, [[np.nan, 0.5, 0.5]]]), c  # an unused vertex, not finite
    if kind == "flat":
        return _box(29, 31, 1, (1.0, 1.0, 1e-6))
    if kind == "long":
        return _box(2, 2, 150, (1e-3, 1e-3, 1.0))
    if kind == "folded":  # coincident coordinates along x: ties in every order
        x, c = _box(9, 8, 7)
        x[:, 0] *= 1.0 + 1e-13
        x[:, 1] = np.round(x[:, 1]) + 1e-9 * x[:, 0]
        return x, c
    if kind == "shuffled":
        x, c = _box(12, 13, 11)
        rng = np.random.default_rng(1)
        pv = rng.permutation(len(x))
        inv = np.empty_like(pv)
        inv[pv] = np.arange(len(x))
        return x[pv] + 0.1 * rng.uniform(-1, 1, x.shape), inv[c][rng.permutation(len(c))].astype(
            np.int32)
    return _star(250)


@pytest.mark.parametrize("rows", [32, 64, 256])
@pytest.mark.parametrize("kind", ["one_cell", "rows_63", "rows_64", "rows_65", "flat", "long",
                                  "folded", "shuffled", "star"])
def test_tiles_assemble_like_the_row_walk(cuda_device, kind, rows):
    import torch
    from dissolve_tp import _lib
    from dissolve_tp.assembler import DeviceMesh
    from dissolve_tp.device import ptr, stream_handle
    xyz, cells = _mesh(kind)
    dm = DeviceMesh(xyz, cells, tile_rows=0)
    rng = np.random.default_rng(2)
    De = torch.from_numpy(rng.uniform(0.5, 2.0, dm.n_cells)).cuda()
    out = []
    # the row walk holds rows of up to about 220 entries; past them tiles of another size
    for r in (0 if dm.max_row_len <= 200 else 128, rows):
        dm.set_tiles(r)
        o = torch.full((dm.nnz + 2,), -7.0, dtype=torch.float64, device="cuda")
        _lib.call("tp_assemble_csr", ctypes.byref(dm.tpm), ptr(De), ptr(De), 20.0, 0,
                  _lib.TP_ASM_FULL, None, ptr(o) + 8, None, stream_handle())
        out.append(o.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    assert out[1][0] == -7.0 and out[1][-1] == -7.0  # nothing written outside the values
    info = dm.tiles_info()
    assert info["n_tiles"] == -(-dm.n_verts // rows)


@pytest.mark.parametrize("rows", [32, 64, 256])
@pytest.mark.parametrize("kind", ["one_cell", "rows_63", "rows_65", "flat", "long", "shuffled",
                                  "star"])
def test_tiles_sum_like_the_row_walk(cuda_device, kind, rows):
    """Lumped diagonal (1 to 4 columns, Dirichlet rows) bit for bit; nodal gradient within
    1e-12 of the largest one (the same sums; the compiler may contract a cell's cofactors
    differently in two kernels), NaN at the same unused vertices."""
    import torch
    from dissolve_tp import _lib
    from dissolve_tp.assembler import DeviceMesh
    from dissolve_tp.device import ptr, stream_handle
    xyz, cells = _mesh(kind)
    dm = DeviceMesh(xyz, cells, tile_rows=0)
    rng = np.random.default_rng(3)
    V = dm.n_verts
    u = torch.from_numpy(rng.uniform(-1.0, 1.0, V)).cuda()
    mask = torch.from_numpy((rng.uniform(0, 1, V) < 0.2).astype(np.uint8)).cuda()
    al = torch.from_numpy(rng.uniform(0, 1, (dm.n_cells, 4))).cuda()
    grads, diags = [], []
    for r in (0, rows):
        dm.set_tiles(r)
        g = torch.full((3 * V + 2,), -7.0, dtype=torch.float64, device="cuda")
        _lib.call("tp_nodal_gradient", ctypes.byref(dm.tpm), None, ptr(u), ptr(g) + 8,
                  stream_handle())
        grads.append(g.cpu().numpy())
        d = []
        for S, ld in ((1, 1), (1, 2), (2, 2), (3, 3), (3, 4), (4, 4)):
            d64 = torch.full((V * ld + 2,), -7.0, dtype=torch.float64, device="cuda")
            d32 = torch.full((V * ld,), -7.0, dtype=torch.float32, device="cuda")
            sh = (ctypes.c_double * 4)(0.5, 50.0, 0.0, 1e-3)
            a = al[:, :ld].contiguous() if S != 2 else None
            _lib.call("tp_lumped_diag", ctypes.byref(dm.tpm), S, ld, ptr(a), sh,
                      ptr(mask) if ld > 1 else None, ptr(d64) + 8, ptr(d32), stream_handle())
            d += [d64.cpu().numpy(), d32.cpu().numpy()]
            assert d[-2][0] == -7.0 and d[-2][-1] == -7.0
        diags.append(d)
    for a, b in zip(*diags):
        assert np.array_equal(a, b)
    assert np.array_equal(np.isnan(grads[0]), np.isnan(grads[1]))
    ref = np.nan_to_num(grads[0])
    assert np.abs(np.nan_to_num(grads[1]) - ref).max() <= 1e-12 * np.abs(ref).max()
    assert grads[1][0] == -7.0 and grads[1][-1] == -7.0

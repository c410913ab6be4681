"""Matrix-free apply from geometry records and, for a mesh without them, from coordinates:
cell counts off the warp and block sizes, cell orders with long, short and no runs of one
vertex, every row width.

Bars: FP64 within 1e-12 (max-norm, relative) of the oracle, FP32 within 2e-5: the bars of
the same comparison at other sizes."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("S,ld", [(1, 1), (1, 2), (2, 2), (3, 4), (4, 4)])
@pytest.mark.parametrize("n,order", [(1, "kuhn"), (3, "shuffled"), (5, "kuhn"), (6, "sorted"),
                                     (19, "kuhn"), (31, "shuffled")])
def test_matfree_routes_match_oracle(cuda_device, n, order, S, ld):
    import torch

    from dissolve_tp import _lib
    from dissolve_tp.assembler import DeviceMesh
    from dissolve_tp.device import ptr, stream_handle
    from dissolve_tp.mesh import kuhn_cube
    m = kuhn_cube(n, 0.2 if n > 1 else 0.0, seed=n)
    rng = np.random.default_rng(n + S)
    cells = np.asarray(m.cells)
    if order == "shuffled":
        cells = cells[rng.permutation(len(cells))]
    elif order == "sorted":  # runs of up to 24 cells with one first vertex
        cells = np.sort(cells, axis=1)
        cells = cells[np.argsort(cells[:, 0], kind="stable")]
    dm = DeviceMesh(m.coords, cells)
    detJ, G, _ = orc.geometry(m.coords, cells)
    De = np.exp(0.3 * rng.standard_normal(len(cells)))
    al = rng.uniform(0, 1, len(cells))
    x = rng.standard_normal((m.n_verts, S))
    ds, sh = np.array([1.0, 0.7, 2.6, 1.3])[:S], np.array([0.5, 0.0, 0.2, 0.1])[:S]
    xd = np.zeros((m.n_verts, ld))
    xd[:, :S] = x
    bare = type(dm.tpm)()
    ctypes.memmove(ctypes.byref(bare), ctypes.byref(dm.tpm), ctypes.sizeof(bare))
    bare.geo = None
    Dd, Ad = torch.from_numpy(De).cuda(), torch.from_numpy(al).cuda()
    dsc, shf = (ctypes.c_double * 4)(*ds), (ctypes.c_double * 4)(*sh)
    for legacy in (0, 1):
        ref = orc.matfree_apply(cells, detJ, G, De, x, 50.0, alpha_cell=al, lumped=legacy,
                                legacy=legacy, diff_scale=ds, shift=sh)
        for mesh in (dm.tpm, bare):
            for fp32, tol in ((0, 1e-12), (1, 2e-5)):
                X = torch.from_numpy(xd).to("cuda", torch.float32 if fp32 else torch.float64)
                Y = torch.full_like(X, 7.0)
                _lib.call("tp_matfree_apply", ctypes.byref(mesh), S, ld, fp32, ptr(Dd), ptr(Ad),
                          dsc, shf, 50.0, legacy, legacy, ptr(X), ptr(Y), stream_handle())
                got = Y.double().cpu().numpy()
                assert np.abs(got[:, :S] - ref).max() <= tol * np.abs(ref).max()
                assert np.all(got[:, S:] == 0.0)

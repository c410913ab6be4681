"""Row tiles of a mesh whose CSR pattern holds more than the cells touch, on one side of the
diagonal only: the entries no cell touches are 0, in CSR and in SELL-32 order, as in the row
walk."""
import ctypes

import numpy as np
import pytest

from test_gpu_tiles_build import _box

pytestmark = pytest.mark.gpu


class _Padded:
    """The mesh with `upper` more columns past each row's diagonal in its pattern."""

    def __init__(self, shape, upper):
        import torch
        from dissolve_tp import _lib
        from dissolve_tp._lib import call
        from dissolve_tp.assembler import DeviceMesh
        from dissolve_tp.device import ptr, stream_handle
        self.dm = dm = DeviceMesh(*_box(*shape), tile_rows=0)
        ip, ix = dm.indptr.cpu().numpy(), dm.indices.cpu().numpy()
        V = dm.n_verts
        rows = [np.union1d(ix[ip[r]:ip[r + 1]], np.arange(r, min(r + upper + 1, V)))
                for r in range(V)]
        self.touched = np.concatenate([np.isin(c, ix[ip[r]:ip[r + 1]])
                                       for r, c in enumerate(rows)])
        self.indptr = torch.from_numpy(
            np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.int32)).cuda()
        self.indices = torch.from_numpy(np.concatenate(rows).astype(np.int32)).cuda()
        self.nnz = int(self.indices.numel())
        self.slots = torch.empty_like(dm.slots)
        self.tpm = t = _lib.TpMesh.from_buffer_copy(dm.tpm)
        t.nnz, t.max_row_len = self.nnz, max(len(c) for c in rows)
        t.indptr, t.indices, t.v2c_slots = ptr(self.indptr), ptr(self.indices), None
        call("tp_incidence_slots", ctypes.byref(t), ptr(self.slots), ptr(dm.flags),
             stream_handle())
        t.v2c_slots = ptr(self.slots)
        self._h = ctypes.c_void_p()

    def tiles(self, rows):
        from dissolve_tp import _lib
        from dissolve_tp.device import stream_handle
        if self._h:
            _lib.lib.tp_tiles_destroy(self._h)
            self._h = ctypes.c_void_p()
        if rows:
            _lib.call("tp_tiles_create", ctypes.byref(self.tpm), rows, stream_handle(),
                      ctypes.byref(self._h))
        self.tpm.tiles = self._h.value


def _assembled(p, S=2):
    import torch
    from dissolve_tp import _lib
    from dissolve_tp.device import ptr, stream_handle
    from dissolve_tp.krylov import SellPattern
    De = torch.from_numpy(np.random.default_rng(2).uniform(0.5, 2.0, p.dm.n_cells)).cuda()
    sell = SellPattern(p.indptr, p.indices)
    # guard values on both sides of every output
    new = lambda n, dt: torch.full((n + 64,), -7.0, dtype=dt, device="cuda")  # noqa: E731
    a, k, s = new(p.nnz, torch.float64), new(p.nnz, torch.float64), new(sell.n_entries,
                                                                        torch.float32)
    d = new(S * p.dm.n_verts, torch.float64)
    _lib.call("tp_assemble_csr", ctypes.byref(p.tpm), ptr(De), ptr(De), 20.0, 0,
              _lib.TP_ASM_FULL, None, ptr(a) + 256, None, stream_handle())
    sh = (ctypes.c_double * 4)(0.5, 50.0, 0.0, 0.0)
    _lib.call("tp_assemble_stiffness_diag", ctypes.byref(p.tpm), ptr(De), S, S, None, sh, None,
              ptr(k) + 256, None, ptr(sell.slice_ptr), ptr(s) + 128, ptr(d) + 256, None,
              stream_handle())
    out = [t.cpu().numpy() for t in (a, k, s, d)]
    for t in out:
        assert np.all(t[:32] == -7.0) and np.all(t[-32:] == -7.0)
    return [t[32:-32] for t in out]


@pytest.mark.parametrize("shape,upper,rows", [((3, 3, 9), 40, 32), ((2, 2, 60), 90, 64),
                                              ((4, 3, 5), 30, 256)])
def test_entries_past_the_cells_are_zero(cuda_device, shape, upper, rows):
    p = _Padded(shape, upper)
    assert not p.touched.all()
    want = _assembled(p)
    p.tiles(rows)
    got = _assembled(p)
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
    assert np.all(got[0][~p.touched] == 0.0) and np.all(got[1][~p.touched] == 0.0)


def test_more_entries_than_a_meshs_tile_can_own(cuda_device):
    """125 entries past each diagonal: tiles of 256 rows own 32,000, more than the six edges
    of each of 4,095 cells."""
    test_entries_past_the_cells_are_zero(cuda_device, (2, 2, 150), 125, 256)

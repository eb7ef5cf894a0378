"""The FP64 visit's loads, which take a record's sectors in an order of the lane's own: records that
start inside a 128-byte line (the ABI asks for 32-byte alignment) and blocks of ragged size give
the oracle's weights, cells and removals bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from helpers import mesh, random_particles
from oppb import _lib as L
from oppb.fempic import DeviceMesh, ParticleSet
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("offset", [0, 4, 8, 12], ids=lambda o: f"{8 * o}B")
@pytest.mark.parametrize("n", [1, 5, 4099])
def test_records_inside_a_line(n, offset):
    hm = mesh()
    dm = DeviceMesh(hm, DEV, mixed=False)
    det = torch.empty(dm.det.numel() + 16, dtype=torch.float64, device=DEV)
    det[offset:offset + dm.det.numel()] = dm.det
    s = L.TetMesh(hm.n_cells, hm.n_nodes, det.data_ptr() + 8 * offset, dm.s.nav, dm.s.c2n, dm.s.ef, None, None)
    pos, p2c = random_particles(hm, n, 40 + n)
    ps = ParticleSet(DEV, n)
    ps.size = n
    ps.pos[:, :n] = torch.from_numpy(np.ascontiguousarray(pos.T)).to(DEV)
    ps.p2c[0, :n] = torch.from_numpy(p2c).to(DEV)
    v = ps.view()
    L.check("move", L.load().oppb_move_f64(C.byref(s), C.byref(v), ps.status.data_ptr(), 4096, None))
    st = ps.status_host()
    lc, ref = np.zeros((n, 4)), p2c.copy()
    O.move(pos, lc, ref, hm.c2c, hm.c_vol, hm.c_det)
    got = ps.host_aos()
    assert st.error == 0 and st.remove_count == int((ref == L.REMOVED_CELL).sum())
    np.testing.assert_array_equal(got["p2c"], ref)
    np.testing.assert_array_equal(got["lc"].view(np.uint64), lc.view(np.uint64))

"""The standalone deposit's cell-ordered rows at their edges: one group of 32 lanes, 32 groups of one,
more than eight groups a warp, invalid and removed cells among valid ones, ragged sizes.  Against the
oracle's sums; two orders of adding the n_k terms of a node differ by at most 2 n_k 2^-53 sum |w|."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from helpers import REMOVED, mesh
from oppb import _lib as L
from oppb.fempic import DeviceMesh, ParticleSet
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 5000])
@pytest.mark.parametrize("kind", ["one", "each", "runs", "nine", "holes"])
def test_deposit_rows(n, kind):
    hm = mesh()
    rng = np.random.default_rng(n)
    i = np.arange(n)
    cell = {"one": np.full(n, 77), "each": (i * 37) % hm.n_cells, "runs": i // 11, "nine": 500 + i % 9,
            "holes": rng.integers(0, hm.n_cells, n)}[kind].astype(np.int32)
    if kind == "holes":
        cell[rng.random(n) < 0.3] = REMOVED
        cell[rng.random(n) < 0.1] = -1
    lc = rng.random((n, 4))
    dm = DeviceMesh(hm, DEV, mixed=False)
    ps = ParticleSet(DEV, n)
    ps.size = n
    ps.lc[:, :n] = torch.from_numpy(np.ascontiguousarray(lc.T)).to(DEV)
    ps.p2c[0, :n] = torch.from_numpy(cell).to(DEV)
    charge = torch.zeros(hm.n_nodes, dtype=torch.float64, device=DEV)
    ws = torch.empty(L.load().oppb_deposit_workspace_bytes(hm.n_nodes), dtype=torch.uint8, device=DEV)
    v = ps.view()
    L.check("deposit", L.load().oppb_deposit_f64(C.byref(dm.s), C.byref(v), charge.data_ptr(), ws.data_ptr(),
                                                 ws.numel(), None))
    ok = (cell >= 0) & (cell < hm.n_cells)
    ref = np.zeros(hm.n_nodes)
    O.deposit(np.ascontiguousarray(lc[ok]), np.ascontiguousarray(cell[ok]), hm.c2n, ref)
    terms = np.bincount(hm.c2n[cell[ok]].ravel(), minlength=hm.n_nodes)
    got = charge.cpu().numpy()
    assert (np.abs(got - ref) <= 2 * terms * 2.0 ** -53 * ref).all()

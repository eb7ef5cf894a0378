"""The hole fill's pairs where its bytes, words and blocks end: sizes around 8, 32 and a block's
16,384 particles, holes at the tail, at the head, alternating and random, against the oracle;
also with fewer pairs than holes would need (every live particle behind the holes moved)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from helpers import REMOVED
from oppb import _lib as L
from oppb.fempic import ParticleSet
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 16383, 16384, 16385, 70001])
@pytest.mark.parametrize("kind", ["tail", "head", "alternate", "random", "most", "all"])
def test_pairs(n, kind):
    rng = np.random.default_rng(n)
    gone = {"tail": np.arange(n) >= n - max(1, n // 5), "head": np.arange(n) < max(1, n // 5),
            "alternate": np.arange(n) % 2 == 0, "random": rng.random(n) < 0.01,
            "most": rng.random(n) < 0.97, "all": np.ones(n, bool)}[kind]
    p2c = np.where(gone, REMOVED, rng.integers(0, 999, n)).astype(np.int32)
    pos, vel, lc = rng.random((n, 3)), rng.random((n, 3)), rng.random((n, 4))
    ps = ParticleSet(DEV, n + 5)
    ps.size = n
    for name, a in (("pos", pos), ("vel", vel), ("lc", lc)):
        getattr(ps, name)[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T)).to(DEV)
    ps.p2c[0, :n] = torch.from_numpy(p2c).to(DEV)
    lib = L.load()
    L.check("bits", lib.oppb_removal_bits(ps.p2c.data_ptr(), n, ps.bits.data_ptr(), None))
    removed = int(gone.sum())
    if removed:
        ws = torch.empty(lib.oppb_hole_fill_workspace_bytes(n, removed), dtype=torch.uint8, device=DEV)
        L.check("hole fill", lib.oppb_hole_fill(n, removed, ps.bits.data_ptr(), ps.capacity, 4, ps.dat_list(),
                                                ws.data_ptr(), ws.numel(), None))
    dats = [pos.copy(), vel.copy(), lc.copy(), p2c.copy()]
    O.hole_fill(n, removed, dats[3], dats)
    left = n - removed
    for name, ref in zip(("pos", "vel", "lc", "p2c"), dats):
        got = getattr(ps, name)[:, :left].T.cpu().numpy().reshape(ref[:left].shape)
        np.testing.assert_array_equal(got, ref[:left], err_msg=name)

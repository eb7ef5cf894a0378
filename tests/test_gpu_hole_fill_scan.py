"""The hole fill on both sides of the line where the emit kernel stops summing the blocks' hole counts
itself and reads a scan of them (1,024 blocks of 16,384 particles), with holes at the head, the
tail, the blocks' edges and all over: the moved values exactly the oracle's."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import REMOVED
from oppb import _lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
BLOCK = 16384
LINE = 1024 * BLOCK


@pytest.mark.parametrize("n", [LINE - 5, LINE, LINE + 1, LINE + 3 * BLOCK + 77])
@pytest.mark.parametrize("kind", ["head", "tail", "edges", "random", "last"])
def test_pairs_at_the_line(n, kind):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    gone = {"head": i < 30000, "tail": i >= n - 30000, "edges": (i % BLOCK < 2) | (i % BLOCK == BLOCK - 1),
            "random": rng.random(n) < 0.003, "last": i == n - 1}[kind]
    p2c = np.where(gone, REMOVED, i % 999).astype(np.int32)
    value = rng.integers(-2 ** 31, 2 ** 31, n).astype(np.int32)
    removed = int(gone.sum())
    d_p2c, d_value = torch.from_numpy(p2c).to(DEV), torch.from_numpy(value).to(DEV)
    bits = torch.zeros((n + 31) // 32, dtype=torch.int32, device=DEV)
    lib = L.load()
    L.check("bits", lib.oppb_removal_bits(d_p2c.data_ptr(), n, bits.data_ptr(), None))
    dats = (L.Dat * 2)(L.Dat(d_p2c.data_ptr(), None, 1, 4), L.Dat(d_value.data_ptr(), None, 1, 4))
    ws = torch.empty(lib.oppb_hole_fill_workspace_bytes(n, removed), dtype=torch.uint8, device=DEV)
    L.check("hole fill", lib.oppb_hole_fill(n, removed, bits.data_ptr(), n, 2, dats, ws.data_ptr(), ws.numel(), None))
    O.hole_fill(n, removed, p2c, [value, p2c])
    left = n - removed
    np.testing.assert_array_equal(d_p2c[:left].cpu().numpy(), p2c[:left])
    np.testing.assert_array_equal(d_value[:left].cpu().numpy(), value[:left])

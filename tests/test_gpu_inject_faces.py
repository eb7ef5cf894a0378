"""The injection's face search where its first guess is right, one off and far off: even, skewed,
single-face and empty-face distributions, fewer particles placed than injected, against
searchsorted (first face j with k < dist[j], the last face if none)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from oppb import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n_faces", [1, 2, 3, 200, 4608])
@pytest.mark.parametrize("kind", ["even", "skewed", "last", "first", "holes", "short"])
def test_faces(n_faces, kind):
    rng = np.random.default_rng(n_faces)
    count = 5003
    share = {"even": np.ones(n_faces), "skewed": np.arange(1, n_faces + 1) ** 3.0,
             "last": np.r_[np.zeros(n_faces - 1), 1.0], "first": np.r_[1.0, np.zeros(n_faces - 1)],
             "holes": (rng.random(n_faces) < 0.3) + 1e-9, "short": np.ones(n_faces)}[kind]
    total = count if kind != "short" else count // 3
    dist = np.floor(np.cumsum(share) / share.sum() * total + 1e-6).astype(np.int32)
    d, p2c = torch.from_numpy(dist).to(DEV), torch.full((count + 7,), -5, dtype=torch.int32, device=DEV)
    inlet = L.Inlet(n_faces, d.data_ptr(), d.data_ptr(), d.data_ptr())
    L.check("faces", L.load().oppb_assign_faces(C.byref(inlet), p2c.data_ptr(), 3, count, None))
    ref = np.minimum(np.searchsorted(dist, np.arange(count), side="right"), n_faces - 1)
    got = p2c.cpu().numpy()
    np.testing.assert_array_equal(got[3:3 + count], ref)
    assert (got[:3] == -5).all() and (got[3 + count:] == -5).all()

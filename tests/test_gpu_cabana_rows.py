"""The CabanaPIC kernel's cell-ordered rows and its queue of face-crossing particles at their edges:
ragged blocks, a cell per particle, all particles in one cell, cells in no order, every particle
crossing several faces, none crossing, and invalid cells among valid ones.  Particles bit-exact
with the oracle, accumulators within 1e-12 of the largest (FP64 sums in another order)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oppb import _lib as L
from oppb.cabana import HexMesh, synthetic_interp
from test_gpu_cabana import _K, _acc_close, _bits_equal, _run_gpu, _run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 256, 1030])
@pytest.mark.parametrize("cells,scale", [("each", 3.0), ("each", 0.0), ("one", 3.0), ("mixed", 0.3)])
def test_rows_and_queue(n, cells, scale, precision):
    mesh = HexMesh(9, 8, 17)
    rng = np.random.default_rng(n)
    interp = synthetic_interp(mesh, 7, e_scale=0.1, b_scale=0.1) if scale else np.zeros((mesh.n_cells, 18))
    p2c = {"each": mesh.interior[rng.permutation(len(mesh.interior))[:n] if n <= len(mesh.interior) else 0],
           "one": np.full(n, mesh.interior[5]), "mixed": rng.choice(mesh.interior[:40], n)}[cells].astype(np.int32)
    pos = rng.uniform(-1.0, 1.0, (n, 3))
    vel = rng.normal(0.0, scale, (n, 3)) if scale else np.zeros((n, 3))
    w, streak = rng.uniform(0.5, 1.5, n), np.zeros((n, 3))
    k = _K(-0.2, (2.3, 1.9, 2.6), -1.0)
    got, st = _run_gpu(mesh, interp, pos, vel, streak, w, p2c, k, precision=precision)
    ref, visits = _run_oracle(mesh, interp, pos, vel, streak, w, p2c, k, precision=precision)
    assert st.error == 0 and int(st.total_visits) == visits
    for name in ("pos", "vel", "streak", "p2c"):
        _bits_equal(got[name], ref[name], name)
    _acc_close(got["acc"], ref["acc"])


def test_invalid_cells_are_left_alone():
    mesh = HexMesh(6, 5, 7)
    rng = np.random.default_rng(3)
    n = 600
    p2c = rng.choice(mesh.interior, n).astype(np.int32)
    bad = rng.random(n) < 0.2
    pos, vel = rng.uniform(-1, 1, (n, 3)), rng.normal(0, 0.5, (n, 3))
    w, streak = np.ones(n), np.zeros((n, 3))
    k = _K(-0.2, (1.4, 0.8, 2.2), -1.0)
    interp = synthetic_interp(mesh, 9)
    ref, _ = _run_oracle(mesh, interp, pos[~bad], vel[~bad], streak[~bad], w[~bad], p2c[~bad], k)
    p2c[bad] = mesh.n_cells + 3
    got, st = _run_gpu(mesh, interp, pos, vel, streak, w, p2c, k)
    assert st.error == L.OPPB_ERR_CELL_RANGE and bad[st.error_index]
    for name, a in (("pos", pos), ("vel", vel), ("streak", streak), ("p2c", p2c)):
        _bits_equal(got[name][bad], a[bad], name)
        _bits_equal(got[name][~bad], ref[name], name)
    _acc_close(got["acc"], ref["acc"])

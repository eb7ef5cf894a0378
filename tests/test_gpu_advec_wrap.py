"""The advection step's wrap and its launch shapes: positions whose quotient by the extent is an integer
or next to one, far outside the extents and on cell edges (in one wave, which divides; the wrap by
reciprocals of larger batches is in test_gpu_advec_grid_form); batches of one item a block, of several, and past the resident blocks.
Positions, directions and cells bit-exact with the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import advec_edge_particles
from oppb import _lib as L
from oppb.advec import AdvecBatchDevice, AdvecMesh
from oracle import advec as OA

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("grid", [True, False], ids=["grid", "records"])
@pytest.mark.parametrize("nx,ny,cw", [(13, 9, 0.7), (61, 61, 1.0), (5, 37, 0.25)])
def test_wrap_next_to_integers(nx, ny, cw, grid):
    m = AdvecMesh(nx, ny, cw)
    rng = np.random.default_rng(nx)
    n = 6000
    ext = np.array(m.extents)
    q = rng.integers(-3, 4, (n, 2)) + rng.choice([0.0, 1e-16, -1e-16, 3e-7, -3e-7, 2e-6, 0.5], (n, 2))
    pos = q * ext
    for _ in range(3):  # a few ulps around the multiples
        step = rng.integers(-1, 2, (n, 2))
        pos = np.where(step > 0, np.nextafter(pos, np.inf), np.where(step < 0, np.nextafter(pos, -np.inf), pos))
    vel, mdir = np.zeros((n, 2)), np.full((n, 2), 7, np.int32)
    p2c = rng.integers(0, m.n_cells, n).astype(np.int32)
    dev = AdvecBatchDevice([m], [n], [0.5], DEV, grid=grid)
    dev.set_instance(0, pos, vel, mdir, p2c)
    dev.zero_status()
    dev.step()
    ref = {"pos": pos.copy(), "mdir": mdir.copy(), "p2c": p2c.copy()}
    visits = OA.steps(ref["pos"], vel, ref["mdir"], ref["p2c"], m.c2c, m.c_pos_ll, 0.5, m.extents, cw, 1)
    got, st = dev.host_instance(0), dev.status_host()
    assert st.error == 0 and int(st.total_visits) == visits
    np.testing.assert_array_equal(got["pos"].view(np.uint64), ref["pos"].view(np.uint64))
    np.testing.assert_array_equal(got["mdir"], ref["mdir"])
    np.testing.assert_array_equal(got["p2c"], ref["p2c"])


@pytest.mark.parametrize("items", [1, 2, 4])
@pytest.mark.parametrize("sides", [[7], [61], [90, 40, 3, 61], [130, 128]], ids=str)
def test_launch_shapes(sides, items):
    """1 item; one item a block; several instances past the resident blocks (chunks of 8 items)."""
    specs = [(AdvecMesh(s, s), 20) for s in sides]
    host = [advec_edge_particles(m, ppc, 0.6, k) for k, (m, ppc) in enumerate(specs)]
    dev = AdvecBatchDevice([m for m, _ in specs], [len(h[3]) for h in host], [0.5] * len(specs), DEV)
    L.set_tuning(advec_items=items)
    try:
        for k, h in enumerate(host):
            dev.set_instance(k, *h)
        for _ in range(3):
            dev.step()
        torch.cuda.synchronize()
    finally:
        L.set_tuning(advec_items=2)
    for k, ((m, _), (pos, vel, mdir, p2c)) in enumerate(zip(specs, host)):
        pos, mdir, p2c = pos.copy(), mdir.copy(), p2c.copy()
        for _ in range(3):
            OA.steps(pos, vel, mdir, p2c, m.c2c, m.c_pos_ll, 0.5, m.extents, 1.0, 1)
        got = dev.host_instance(k)
        np.testing.assert_array_equal(got["pos"].view(np.uint64), pos.view(np.uint64))
        np.testing.assert_array_equal(got["mdir"], mdir)
        np.testing.assert_array_equal(got["p2c"], p2c)


def test_invalid_cell_keeps_its_direction():
    m = AdvecMesh(8, 8)
    pos, vel, mdir, p2c = advec_edge_particles(m, 4, 0.3, 1)
    mdir[:] = 5
    p2c[17] = 64
    dev = AdvecBatchDevice([m], [len(p2c)], [0.5], DEV)
    dev.set_instance(0, pos, vel, mdir, p2c)
    dev.zero_status()
    dev.step()
    got, st = dev.host_instance(0), dev.status_host()
    assert st.error == L.OPPB_ERR_CELL_RANGE and st.error_index == 17
    assert (got["mdir"][17] == 5).all() and got["p2c"][17] == 64
    assert (np.delete(got["mdir"], 17, 0) == 0).all()

"""The kernels for batches of grids only (oppb_advec_step_grid, oppb_advec_move_grid) against the general
ones on the same state, bit for bit: sizes of one item a block and past the resident blocks, every
number of items a pass, with and without the global move, quotients at and extents past the limits of
the wrap by a reciprocal, and an instance without a grid, which they refuse particle by particle."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from helpers import advec_edge_particles
from oppb import _lib as L
from oppb.advec import AdvecBatchDevice, AdvecMesh

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _pair(meshes, host, dts, dh=None):
    out = []
    for _ in range(2):
        d = AdvecBatchDevice(meshes, [len(h[3]) for h in host], dts, DEV)
        for k, h in enumerate(host):
            d.set_instance(k, *h)
        if dh:
            d.enable_direct_hop(dh)
        d.zero_status()
        out.append(d)
    return out


def _call(d, what: str, general: bool) -> None:
    fn = getattr(d.lib, f"oppb_advec_{what}" + ("" if general else "_grid"))
    L.check(what, fn(C.byref(d.batch), d.status.data_ptr(), 4096, None))


def _same(a, b) -> None:
    torch.cuda.synchronize()
    for name in ("pos", "mdir", "p2c", "status"):
        x, y = getattr(a, name), getattr(b, name)
        assert torch.equal(x.view(torch.int64) if x.dtype == torch.float64 else x,
                           y.view(torch.int64) if y.dtype == torch.float64 else y), name


@pytest.mark.parametrize("dh", [None, 0.7])
@pytest.mark.parametrize("items", [1, 2, 4])
@pytest.mark.parametrize("sides", [[7], [61], [130, 3, 97, 128]], ids=str)
def test_equal_to_the_general_kernel(sides, items, dh):
    meshes = [AdvecMesh(s, max(2, s // 2)) for s in sides]
    host = [advec_edge_particles(m, 23, 0.6, k) for k, m in enumerate(meshes)]
    a, b = _pair(meshes, host, [0.5] * len(meshes), dh)
    L.set_tuning(advec_items=items)
    try:
        for _ in range(3):
            _call(a, "step", False)
            _call(b, "step", True)
        for d in (a, b):
            d.update_pos()
            _call(d, "move", d is b)
    finally:
        L.set_tuning(advec_items=2)
    _same(a, b)


@pytest.mark.parametrize("cw,dh", [(1e-320, None)] + [(c, d) for c in (1e-300, 3e-39, 1e-30, 1e37, 1e39, 1e300)
                                                      for d in (None, 1.0)])
def test_extents_past_fp32(cw, dh):
    """The wrap by a reciprocal that the block keeps, or with the global move one of its own, whatever the
    extent's size.  Without the global move the cells are invalid, so that nothing walks; with it the
    walks start from the grid's cells where it has any at that size."""
    m = AdvecMesh(60, 60, cw)
    rng = np.random.default_rng(1)
    n = 1300 * 256  # more passes than resident blocks
    pos, vel = rng.uniform(-0.2, 1.2, (n, 2)) * m.extents[0], rng.normal(0.0, 0.3, (n, 2)) * cw
    host = [(pos, vel, np.ones((n, 2), np.int32), np.full(n, m.n_cells, np.int32))]
    a, b = _pair([m], host, [0.5], dh and dh * cw)
    assert a.all_grid
    _call(a, "step", False)
    _call(b, "step", True)
    torch.cuda.synchronize()
    assert torch.equal(a.pos.view(torch.int64), b.pos.view(torch.int64))
    assert torch.equal(a.p2c, b.p2c) and torch.equal(a.mdir, b.mdir)
    a.update_pos()  # keeps reciprocals too, where the general step divides
    _call(b, "step", True)
    torch.cuda.synchronize()
    assert torch.equal(a.pos.view(torch.int64), b.pos.view(torch.int64))


@pytest.mark.parametrize("dh", [None, 0.7])
@pytest.mark.parametrize("nx,ny,cw", [(13, 9, 0.7), (61, 61, 1.0), (5, 37, 0.25)])
def test_quotients_next_to_integers(nx, ny, cw, dh):
    """Multiples of the extents, a few ulps and up to 2^-18 around them, where the divide decides or takes
    over from the reciprocal, in batches of more than one wave (one wave always divides)."""
    m = AdvecMesh(nx, ny, cw)
    rng = np.random.default_rng(nx)
    n = 1300 * 256
    away = [0.0, 1e-16, -1e-16, 3e-7, -3e-7, 2.0 ** -20, -2.0 ** -20, 2e-6, -3e-6, 0.5]
    pos = (rng.integers(-3, 4, (n, 2)) + rng.choice(away, (n, 2))) * np.array(m.extents)
    for _ in range(3):
        step = rng.integers(-1, 2, (n, 2))
        pos = np.where(step > 0, np.nextafter(pos, np.inf), np.where(step < 0, np.nextafter(pos, -np.inf), pos))
    host = [(pos, np.zeros((n, 2)), np.full((n, 2), 7, np.int32), rng.integers(0, m.n_cells, n).astype(np.int32))]
    a, b = _pair([m], host, [0.5], dh)
    _call(a, "step", False)
    _call(b, "step", True)
    _same(a, b)
    c, _ = _pair([m], host, [0.5])
    c.update_pos()
    torch.cuda.synchronize()
    assert torch.equal(c.pos.view(torch.int64), b.pos.view(torch.int64))


@pytest.mark.parametrize("ppc", [3, 90])
def test_an_instance_without_a_grid_is_refused(ppc):
    m = AdvecMesh(70, 60)
    host = [advec_edge_particles(m, ppc, 0.3, 1)]
    a, _ = _pair([m], host, [0.5])
    rec = AdvecBatchDevice([m], [len(host[0][3])], [0.5], DEV, grid=False)
    rec.set_instance(0, *host[0])
    assert a.all_grid and not rec.all_grid
    before = rec.p2c.clone()
    rec.zero_status()
    _call(rec, "step", False)
    st = rec.status_host()
    assert st.error == L.OPPB_ERR_CELL_RANGE and st.total_visits == 0
    assert torch.equal(rec.p2c, before)

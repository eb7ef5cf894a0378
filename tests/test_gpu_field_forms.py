"""The Newton step on K by diagonals (one cluster up to 18,432 unknowns, one block per SM above)
against the same step on K as CSR, which the general kernel takes, around the edges of the split
of rows over blocks and threads.  Both run the same CG on bit-identical products and differ in
the order of the dot products and of the F1 / J-diagonal atomics only: the iteration counts agree
to one and the potentials to the CG's tolerance (1e-10 of ||B||, amplified by the condition of
these boxes to below 1e-8)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oppb.fempic import HostMesh
from oppb.field import FieldConstants, FieldDevice, boundary_potential

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
UNIT = dict(n0=1.0, phi0=0.0, kte=100.0, qe=1.0, eps0=1.0)

# (nx, ny, nz): three 64-row blocks; 5 rows past 16 x 64; a wide window; the last mesh of the cluster
# form and the first of the grid form; several rows a thread with K partly streamed.
DIMS = [(4, 4, 8), (6, 6, 22), (40, 9, 12), (16, 16, 64), (17, 17, 60), (44, 44, 150)]


@pytest.mark.parametrize("dims", DIMS, ids=str)
def test_diagonal_form_equals_csr_form(dims):
    hm = HostMesh(*dims, 1.0, 1.0, 4.0, solve_field=False)
    bnd = boundary_potential(hm.n_type, 1.0, 0.0)
    fd = FieldDevice(hm, DEV, bnd)
    assert len(fd.dia_off) > 0
    ion = torch.from_numpy(np.random.default_rng(3).random(hm.n_nodes) * 2.0).to(DEV)
    c = FieldConstants(**UNIT)
    out = []
    for by_diagonals in (False, True):
        fd.set_diagonal_form(by_diagonals)
        fd.d.zero_()
        fd.f1.zero_()
        for _ in range(2):  # F1 accumulates and D moves on
            pot = fd.solve(ion, c).clone()
        st = fd.status_host()
        assert st.converged == 1 and st.resid * st.b_norm <= max(1e-10 * st.b_norm, 1e-10) * (1 + 1e-9)
        out.append((pot, fd.d[:fd.neq].clone(), fd.f1[:fd.neq].clone(), st.iterations, st.b_norm))
    (p0, d0, f0, i0, b0), (p1, d1, f1, i1, b1) = out
    assert abs(i0 - i1) <= 1
    assert abs(b0 - b1) <= 1e-6 * b0  # the second step's B holds what the first one's CG left
    assert float((f0 - f1).abs().max()) <= 1e-12 * float(f0.abs().max())
    for a, b in ((p0, p1), (d0, d1)):
        assert float((a - b).abs().max()) <= 1e-8 * float(a.abs().max())


@pytest.mark.parametrize("dims", [(6, 6, 12), (20, 20, 64)], ids=str)
def test_no_iterations_leaves_d(dims):
    hm = HostMesh(*dims, 1.0, 1.0, 4.0, solve_field=False)
    fd = FieldDevice(hm, DEV, boundary_potential(hm.n_type, 1.0, 0.0))
    start = torch.from_numpy(np.random.default_rng(5).normal(0.0, 1.0, fd.neq)).to(DEV)
    fd.d[:fd.neq] = start
    fd.solve(torch.ones(hm.n_nodes, dtype=torch.float64, device=DEV), FieldConstants(**UNIT, max_iter=0))
    st = fd.status_host()
    assert st.iterations == 0 and st.converged == 0
    assert torch.equal(fd.d[:fd.neq], start)

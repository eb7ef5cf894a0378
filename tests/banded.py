"""Banded systems for oppb_field_solve made directly through its ABI, without a mesh: K symmetric with
the given positive offsets, every row's diagonal at least 1 above the sum of its other entries'
magnitudes, so that the smallest eigenvalue of J is at least 1."""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from oppb import _lib as L


class Banded:
    def __init__(self, neq: int, offsets, device, seed: int = 0):
        rng = np.random.default_rng(seed)
        offs = np.array(sorted({-o for o in offsets} | {0} | set(offsets)), np.int64)
        dia = np.zeros((len(offs), neq))
        for o in offsets:
            w = -rng.random(neq - o)
            dia[np.searchsorted(offs, o), :neq - o] = w
            dia[np.searchsorted(offs, -o), o:] = w
        dia[np.searchsorted(offs, 0)] = np.abs(dia).sum(0) + 1.0 + rng.random(neq)
        cols = np.arange(neq)[:, None] + offs
        mask = (cols >= 0) & (cols < neq)
        n_nodes = max(neq, 4)
        n2e = np.full(n_nodes, -1, np.int32)
        n2e[:neq] = np.arange(neq)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)  # noqa: E731
        self.neq, self.offs, self.device = neq, offs, device
        self.lib = L.load()
        # one cell whose integrals change F1 and J's diagonal of its four unknowns a little
        self.arrays = dict(n2e=t(n2e), c2n=t(np.arange(4, dtype=np.int32)), det_j=t(np.full(1, 1e-3)),
                           bnd=t(np.zeros(n_nodes)), rowptr=t(np.r_[0, np.cumsum(mask.sum(1))].astype(np.int64)),
                           col=t(cols[mask].astype(np.int32)), val=t(dia.T[mask]), f0=t(rng.normal(0.0, 1.0, neq)),
                           dia=t(dia))
        f = lambda n: torch.zeros(n, dtype=torch.float64, device=device)  # noqa: E731
        self.d, self.f1, self.pot, self.ion, self.status = f(neq), f(neq), f(n_nodes), f(n_nodes), f(3)
        self.work = f(int(self.lib.oppb_field_work_doubles(neq)))

    def struct(self, diagonals: bool) -> L.FieldDevice:
        p = {k: v.data_ptr() for k, v in self.arrays.items()}
        s = L.FieldDevice(len(self.pot), 1, self.neq, 0, p["n2e"], p["c2n"], p["det_j"], p["bnd"], p["rowptr"], p["col"],
                          p["val"], p["f0"], self.d.data_ptr(), self.f1.data_ptr(), self.work.data_ptr())
        if diagonals:
            s.n_diag, s.dia_val = len(self.offs), p["dia"]
            for j, o in enumerate(self.offs):
                s.dia_off[j] = int(o)
        return s

    def launch(self, diagonals: bool = True, max_iter: int = 4000, stream=None, d0: float = 0.0,
               max_polls: int | None = None, no_cluster: bool = False) -> int:
        """One solve from D = d0 and F1 = 0; returns the status code of the call."""
        with torch.cuda.stream(stream):
            self.d.fill_(d0)
            self.f1.zero_()
        c = L.FieldConsts(1.0, 0.0, 100.0, 1.0, 1.0, 1e-10, 1e-10, max_iter, 0)
        args = [C.byref(self.struct(diagonals)), C.byref(c), self.ion.data_ptr(), self.pot.data_ptr(),
                self.status.data_ptr()]
        s = stream.cuda_stream if stream is not None else None
        if max_polls is None and not no_cluster:
            return self.lib.oppb_field_solve(*args, s)
        options = L.FieldOptions(1 << 20 if max_polls is None else max_polls, int(no_cluster))
        return self.lib.oppb_field_solve_ex(*args, C.byref(options), s)

    def solve(self, diagonals: bool = True, **kw) -> tuple[torch.Tensor, L.FieldStatus]:
        L.check("oppb_field_solve", self.launch(diagonals, **kw))
        torch.cuda.synchronize(self.device)
        return self.d.clone(), L.FieldStatus.from_buffer_copy(self.status.cpu().numpy().tobytes())

    def assert_close(self, a, b) -> None:
        """Two solves (d, status) of this system: both residuals are at most max(rtol ||B||, atol) and
        the smallest eigenvalue of J is at least 1, so the solutions lie within twice that
        (a twentieth added for the recurrences' drift); the iteration counts within one."""
        (d0, s0), (d1, s1) = a, b
        assert s0.converged == 1 and s1.converged == 1
        assert abs(s0.iterations - s1.iterations) <= 1
        assert float((d0 - d1).norm()) <= 2.1 * max(1e-10 * s0.b_norm, 1e-10)

"""Field systems of different size solved in turn and from two host threads at once: kernels that they
share take more shared memory for the one than for the other."""
from __future__ import annotations

import ctypes as C
import threading

import pytest
import torch

from banded import Banded
from oppb import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
# two systems of one row a thread for each form: one block per SM, one cluster
PAIRS = {"grid": ((90001, [1, 2000, 4000]), (20001, [1])), "cluster": ((9001, [1, 2000, 4000]), (3001, [1]))}


@pytest.mark.parametrize("form", PAIRS)
def test_in_turn(form):
    big, small = (Banded(n, o, DEV) for n, o in PAIRS[form])
    first = big.solve()
    big.assert_close(first, big.solve(diagonals=False))
    small.assert_close(small.solve(), small.solve(diagonals=False))
    assert torch.equal(big.solve()[0], first[0])


@pytest.mark.parametrize("form", PAIRS)
def test_two_threads(form):
    systems = [Banded(n, o, DEV) for n, o in PAIRS[form]]
    whole = [b.solve()[0] for b in systems]
    torch.cuda.synchronize()
    failed, go = [], threading.Barrier(2)

    def solves(b: Banded) -> None:  # on one stream, so that the solves do not share the SMs
        s, c = b.struct(True), L.FieldConsts(1.0, 0.0, 100.0, 1.0, 1.0, 1e-10, 1e-10, 0, 0)
        args = (C.byref(s), C.byref(c), b.ion.data_ptr(), b.pot.data_ptr(), b.status.data_ptr(), None)
        go.wait()
        for _ in range(3000):
            rc = b.lib.oppb_field_solve(*args)
            if rc:
                failed.append(rc)

    threads = [threading.Thread(target=solves, args=(b,)) for b in systems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == []
    for b, d in zip(systems, whole):
        assert torch.equal(b.solve()[0], d)

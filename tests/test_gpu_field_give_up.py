"""The CG's bounded waits run out: with no poll no block gets through its first reduction, with a few some
do and some do not.  Either the whole step is taken, converged, or D and the potentials of D stay;
a solve with the usual bound then works in the same work space."""
from __future__ import annotations

import pytest
import torch

from banded import Banded
from oppb import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("max_polls", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("neq", [18433, 100001])
def test_no_part_of_a_step(neq, max_polls):
    b = Banded(neq, [1, 130], DEV)
    whole = b.solve(d0=0.25)
    given_up = 0
    for _ in range(20):
        d, st = b.solve(d0=0.25, max_polls=max_polls)
        if st.converged:
            assert torch.equal(d, whole[0])
        else:
            given_up += 1
            assert (d == 0.25).all()
        assert torch.equal(b.pot[:neq], d)
    assert given_up == 20 if max_polls == 0 else True
    again = b.solve(d0=0.25)
    assert again[1].converged == 1 and torch.equal(again[0], whole[0])


def test_negative_bound_is_refused():
    b = Banded(20000, [1], DEV)
    assert b.launch(max_polls=-1) == L.OPPB_ERR_ARG

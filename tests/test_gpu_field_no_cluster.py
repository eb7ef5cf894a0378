"""Small systems by diagonals where no cluster of blocks can be placed: from 64 unknowns on the blocks poll
(four launches a solve), below the general kernel takes them (one); both give the cluster's solution
and the general kernel's."""
from __future__ import annotations

import pytest
import torch

from banded import Banded

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("neq", [1, 63, 64, 65, 129, 577, 4719, 18432])
def test_without_a_cluster(neq):
    b = Banded(neq, [o for o in (1, 30) if o < neq], DEV)
    before = b.lib.oppb_kernel_launches()
    got = b.solve(no_cluster=True)
    assert b.lib.oppb_kernel_launches() - before == (4 if neq >= 64 else 1)
    b.assert_close(got, b.solve())
    b.assert_close(got, b.solve(diagonals=False))
    assert torch.equal(got[0], b.solve(no_cluster=True)[0])

"""The cluster form of the CG while other work holds SMs and shared memory, so that its blocks start at
different times: last blocks of one row and full ones, solved over and over beside matrix products on
a second stream.  Every solve gives the same bits, and the general kernel's solution."""
from __future__ import annotations

import pytest
import torch

from banded import Banded

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("neq", [1, 64, 65, 577, 961, 1025, 18432])
def test_blocks_that_start_late(neq):
    b = Banded(neq, [o for o in (1, 30) if o < neq], DEV)
    alone = b.solve()
    b.assert_close(alone, b.solve(diagonals=False))
    x = torch.randn(2048, 2048, device=DEV)
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(40):
        with torch.cuda.stream(side):
            x @ x
        assert b.launch(stream=main) == 0
        main.synchronize()
        assert torch.equal(b.d, alone[0])
    torch.cuda.synchronize()

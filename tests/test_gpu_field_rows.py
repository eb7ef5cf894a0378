"""The rows a thread of the CG's one-block-per-SM form, two to eight, at the first and last sizes of each, and
the systems by diagonals past it, which the general kernel takes (one launch a solve instead of
four): more rows than eight a thread, and a window of p wider than a block's shared memory.  Against
the solve of the same system as CSR."""
from __future__ import annotations

import pytest
import torch

from banded import Banded

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
PER_ROW = 148 * 640  # unknowns a row a thread: B200's SMs, the form's most threads


@pytest.mark.parametrize("neq", [PER_ROW + 1, 2 * PER_ROW + 1, 4 * PER_ROW + 1, 5 * PER_ROW + 1, 6 * PER_ROW,
                                 6 * PER_ROW + 1, 7 * PER_ROW + 1, 8 * PER_ROW])
def test_rows_a_thread(neq):
    b = Banded(neq, [1, 517], DEV)
    before = b.lib.oppb_kernel_launches()
    got = b.solve()
    assert b.lib.oppb_kernel_launches() - before == 4
    b.assert_close(got, b.solve(diagonals=False))


@pytest.mark.parametrize("neq,offsets,launches", [(8 * PER_ROW + 1, [1, 517], 1), (60000, [1, 13000], 4),
                                                  (60000, [1, 15000], 1), (15000, [1, 14500], 1)], ids=str)
def test_past_the_form(neq, offsets, launches):
    b = Banded(neq, offsets, DEV)
    before = b.lib.oppb_kernel_launches()
    got = b.solve()
    assert b.lib.oppb_kernel_launches() - before == launches
    b.assert_close(got, b.solve(diagonals=False))

"""FemPIC.step through the one native call (oppb_step_begin) against the same step made of the single
entry points (the timed form): the same records and particle bits for every form of the push, the
deposit and the seed, and the move's errors raised the same way."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import mesh
from oppb._lib import OppbError
from oppb.fempic import FemPIC, StepTimes, injection_randoms, randoms_to_device

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
FORMS = {"f64": {}, "mixed": dict(precision="mixed"), "separate push": dict(fused_push=False),
         "mixed, separate push": dict(precision="mixed", fused_push=False), "loops": dict(fused_deposit=False),
         "direct hop": dict(direct_hop=0.05), "direct hop, mixed": dict(direct_hop=0.05, precision="mixed"),
         "sorted": dict(fill="Sort_Periodic", fill_period=3)}


@pytest.mark.parametrize("form", FORMS)
def test_step_equals_its_parts(form):
    sims = [FemPIC(mesh(), DEV, inject_per_step=700, dt=0.05, **FORMS[form]) for _ in range(2)]
    for k in range(12):
        n = 700 if k != 5 else 210  # one odd-sized injection
        t = randoms_to_device(injection_randoms(3, k, 700, 0.1), DEV)[:, :n]
        records = [sims[0].step(t), sims[1].step(t, timers=StepTimes())]
        assert records[0] == records[1]
    a, b = (s.parts.host_aos() for s in sims)
    for name in a:
        np.testing.assert_array_equal(a[name], b[name], err_msg=name)
    q, r = sims[0].node_charge.cpu().numpy(), sims[1].node_charge.cpu().numpy()
    assert np.abs(q - r).max() <= 1e-12 * max(1.0, np.abs(r).max())


def test_hop_limit_is_raised():
    sim = FemPIC(mesh(), DEV, inject_per_step=700, dt=0.8, max_hops=2)
    with pytest.raises(OppbError, match="hop limit"):
        for k in range(3):
            sim.step(randoms_to_device(injection_randoms(3, k, 700, 0.1), DEV))

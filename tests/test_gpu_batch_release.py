"""A plan's captured graph does not outlive the workspace it was captured with."""

import numpy as np
import pytest
import torch

from idi_b200 import _native as nat
from idi_b200.simulation import _core
from idi_b200.simulation.batch import BatchPlan
from tests.helpers import K64, atoms, rng, sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_plan_runs_again_after_release(graph):
    g = rng(31)
    counts = [5000, 300]
    at = torch.from_numpy(np.concatenate([atoms(sphere(g, c, 0.01), g.uniform(0, 6.28, c)) for c in counts])).cuda()
    plan = BatchPlan(counts, _core.make_geom([64, 64], 75.0, 1e5, K64, flags=nat.NF), nat.SPLIT, nat.OUT_C64,
                     autotune=False, graph=graph)
    first = plan.run(at).clone()
    size = _core.WORKSPACES.peek(plan.device, plan._role).numel()
    torch.cuda.synchronize()
    _core.release()
    # what the workspace was is others' memory now, and stays as it is
    others = [torch.full((size,), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
    for _ in range(2):
        assert torch.equal(plan.run(), first)
    plan.check()
    assert _core.WORKSPACES.peek(plan.device, plan._role).numel() >= size
    assert all(bool((o == 7).all()) for o in others)
    plan.close()

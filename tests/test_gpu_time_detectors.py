"""Time path on a detector whose pixel count is at the work queue's limits."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from helpers import K64  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402


def test_time_forward_on_two_to_the_30_pixels():
    """Every CTA claims one share past the end, so the queue counts to twice the pixels, 2^31: more
    than a signed counter holds.  One emitter: tau / 2 at every pixel, none left out."""
    side, tau = 32768, 2.0
    at = torch.tensor([[0.001, -0.002, 0.003, 0.5]], dtype=torch.float64, device="cuda")
    t = torch.zeros(1, dtype=torch.float64, device="cuda")
    out = torch.full((side, side), float("nan"), dtype=torch.float64, device="cuda")
    _core.time_forward(at, t, _core.make_geom([side, side], 5.0, 1e6, K64), 0.3, tau, out=out)
    _core.workspace_error(role="time")
    assert float(out.sub_(tau / 2).abs_().max()) < 1e-15
    del out
    torch.cuda.empty_cache()

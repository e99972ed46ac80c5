"""Radial correlator from several streams: each call has a workspace of its own."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from idi_b200 import _native as nat  # noqa: E402
from idi_b200.reconstruction import _geometry  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402


def test_radial_calls_on_two_streams(monkeypatch):
    """A detector whose rows mirror and one whose rows do not, in turn on two streams: what one
    call keeps in its workspace is not the other's (by address, and by the results)."""
    shape, qmax = (40, 64), 50
    g = np.random.default_rng(3)
    lib, seen = nat.load(), []
    call = lib.idiwf_qcorr_radial

    class Spy:
        def __getattr__(self, name):
            return getattr(lib, name)

        def idiwf_qcorr_radial(self, *args):
            seen.append(args[7].value)
            return call(*args)

    monkeypatch.setattr(_core.nat, "load", lambda: Spy())
    streams = [torch.cuda.Stream() for _ in range(2)]
    jobs, outs = [], []
    for i in range(8):
        q = _geometry.q_rows(shape, 200.0, *((None, None) if i % 2 else (19.5, None)))
        imgs = g.exponential(1.0, (2,) + shape).astype(np.float32)
        jobs.append((q, imgs, torch.from_numpy(q).cuda(), torch.from_numpy(imgs).cuda()))
    torch.cuda.synchronize()
    for i, (_, _, d_q, d_imgs) in enumerate(jobs):
        with torch.cuda.stream(streams[i % 2]):
            outs.append(_core.qcorr_radial(d_q, d_imgs, qmax))
    torch.cuda.synchronize()
    assert not set(seen[::2]) & set(seen[1::2])
    for (q, imgs, _, _), out in zip(jobs, outs):
        np.testing.assert_allclose(out.cpu().numpy(), oracle.qcorr_radial(q, imgs, qmax), rtol=1e-11, atol=1e-9)

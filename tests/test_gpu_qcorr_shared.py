"""Radial correlator: walks shared by the images of a stack and by mirror rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from idi_b200.reconstruction import _geometry  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402


@pytest.mark.parametrize("images", [1, 2, 3, 5])
@pytest.mark.parametrize("shape,qmax,centre", [
    ((1, 40), 15, (None, None)),     # one row: no mirror
    ((2, 33), 20, (None, None)),
    ((31, 50), 24, (None, None)),    # odd rows: half-integer centre, still mirrored
    ((48, 35), 511, (None, None)),   # odd columns, more bins than the detector reaches
    ((40, 64), 300, (20.0, 11.0)),   # mirrored rows, columns off centre
    ((40, 64), 64, (19.5, None)),    # rows off centre
    ((300, 12), 121, (None, None)),  # enough row pairs for two target rows per CTA, the last alone
])
def test_radial_shared_walks_vs_oracle(images, shape, qmax, centre):
    """The runs are the reference's, so only the FP64 additions' order differs (1e-11)."""
    g = np.random.default_rng(images + shape[0])
    imgs = g.exponential(1.0, (images,) + shape).astype(np.float32)
    q = _geometry.q_rows(shape, 200.0, *centre)
    out = _core.qcorr_radial(torch.from_numpy(q).cuda(), torch.from_numpy(imgs).cuda(), qmax).cpu().numpy()
    np.testing.assert_allclose(out, oracle.qcorr_radial(q, imgs, qmax), rtol=1e-11, atol=1e-9)


def test_radial_q_that_only_almost_mirrors():
    """One q value off by an ulp: the rows are walked on their own."""
    g = np.random.default_rng(9)
    shape = (36, 44)
    imgs = g.exponential(1.0, (2,) + shape).astype(np.float32)
    q = _geometry.q_rows(shape, 150.0).copy()
    i = 30 * shape[1] + 7
    q[i, 1] = np.nextafter(q[i, 1], np.float32(1e9))
    out = _core.qcorr_radial(torch.from_numpy(q).cuda(), torch.from_numpy(imgs).cuda(), 40).cpu().numpy()
    np.testing.assert_allclose(out, oracle.qcorr_radial(q, imgs, 40), rtol=1e-11, atol=1e-9)

"""Charge sharing on the tiled kernel: edges of its 32 x 32 tiles and of its photon chunks."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402


@pytest.mark.parametrize("shape", [(1, 1), (31, 32), (33, 65), (100, 37)])
@pytest.mark.parametrize("s,ns", [(0.3, 0.0), (0.9, 0.2), (1.9, 0.0)])
@pytest.mark.parametrize("mean", [0.05, 2.0, 30.0])
def test_tiles_and_chunks_vs_oracle(shape, s, ns, mean):
    """Sparse images (no photons in most regions) to 30 photons a pixel (over a hundred chunks of a
    region), against the oracle's sums in the same order; the factors differ in erf's last bits."""
    g = np.random.default_rng(int(100 * s) + shape[0])
    counts = g.poisson(mean, (2,) + shape).astype(np.int64)
    counts[0, -1, -1] = 700  # one pixel with more photons than a chunk holds
    out = _core.chargesharing(torch.from_numpy(counts).cuda(), s, ns, key=(5, 6), stream=3).cpu().numpy()
    ref = np.stack([oracle.chargesharing(counts, s, ns, key=(5, 6), stream=3)[b] for b in range(2)])
    np.testing.assert_allclose(out, ref, rtol=1e-12, atol=1e-15)


@pytest.mark.parametrize("s,ns,mean", [(0.5, 0.0, 0.05), (0.9, 0.2, 1.0)])
def test_tall_tiles_vs_oracle(s, ns, mean):
    """Enough 32 x 32 tiles for the tall form (a full wave of them), the last row of tiles one pixel high."""
    counts = np.random.default_rng(17).poisson(mean, (2, 97, 3000)).astype(np.int32)
    out = _core.chargesharing(torch.from_numpy(counts).cuda(), s, ns, key=(5, 6), stream=3).cpu().numpy()
    np.testing.assert_allclose(out, oracle.chargesharing(counts, s, ns, key=(5, 6), stream=3), rtol=1e-12, atol=1e-15)

"""Band-limited evaluation at its edges: batches over several launches, images beside
others, differentiation outputs of cut objects, large counts, tuning, large detectors."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from helpers import K64, atoms, rng, sphere  # noqa: E402
from idi_b200 import _native as nat  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402


def _image(g, n, r):
    return atoms(sphere(g, n, r), g.uniform(0, 2 * np.pi, n))


def _forward(at, off, geom, out, precision=nat.SPLIT, **kw):
    t = torch.from_numpy(np.ascontiguousarray(at)).cuda()
    E = _core.forward(t, off, geom, precision, out, **kw).cpu().numpy()
    _core.workspace_error()
    return E


@pytest.mark.parametrize("n_images", [513, 520])
def test_a_launch_of_empty_images(n_images):
    """Of more than 512 images, one large enough for cells and a last launch without emitters."""
    g = rng(20)
    at = _image(g, 6000, 0.01)
    geom = _core.make_geom([64, 64], 75.0, 1e5, K64)
    off = np.full(n_images + 1, len(at), np.int64)
    off[0] = 0
    E = _forward(at, off, geom, nat.OUT_C64)
    assert np.all(E[1:] == 0)
    assert np.array_equal(E[0], _forward(at, [0, len(at)], geom, nat.OUT_C64)[0])


@pytest.mark.parametrize("ndet,spec", [
    # (emitters, radius): in each, an image whose cut would be limited by buffers sized for
    # it alone, beside a larger one
    ([512, 512], [(5000, 0.015), (20000, 0.015)]),  # one grid alone, 72 cells beside
    ([881, 941], [(8169, 0.0076), (20000, 0.01)]),  # to the image's nodes
    ([170, 157], [(7418, 0.107), (100000, 0.1)]),   # direct alone, cells to the pixels beside
])
def test_cut_does_not_depend_on_the_batch(ndet, spec):
    """An image of a batch takes the cut that it takes alone: the pairs formed add up, and the
    float32 intensities are the same."""
    g = rng(21)
    imgs = [_image(g, n, r) for n, r in spec]
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, flags=nat.NF)
    off = np.concatenate([[0], np.cumsum([n for n, _ in spec])])
    E = _forward(np.concatenate(imgs), off, geom, nat.OUT_I32)
    pairs = _core.evaluated_pairs()
    for b, a in enumerate(imgs):
        one = _forward(a, [0, len(a)], geom, nat.OUT_I32)[0]
        pairs -= _core.evaluated_pairs()
        # (another order of the cells' FP64 additions moves a float32 by at most an ulp)
        np.testing.assert_allclose(one, E[b], rtol=1.2e-7, atol=0)
    assert pairs == 0


@pytest.mark.parametrize("out", [nat.OUT_C128, nat.OUT_C64, nat.OUT_I64])
@pytest.mark.parametrize("ndet,spec", [
    ([512, 512], [(5000, 0.015), (20000, 0.015)]),
    ([300, 301], [(4096, 0.02), (9000, 0.04), (12001, 0.01), (30000, 0.03)]),
    ([64, 80], [(100000, 0.15), (5000, 0.01), (70001, 0.12)]),  # to the pixels and to nodes
])
def test_images_cut_into_cells_have_the_bits_they_have_alone(ndet, spec, out):
    """The cells' sums are added on a grid on which FP64 additions are exact, so the bits do not
    depend on how the batch's cells were shared out."""
    g = rng(22)
    imgs = [_image(g, n, r) for n, r in spec]
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, flags=nat.NF)
    off = np.concatenate([[0], np.cumsum([n for n, _ in spec])])
    E = _forward(np.concatenate(imgs), off, geom, out)
    assert _core.evaluated_pairs() < off[-1] * ndet[0] * ndet[1] / 2
    for b, a in enumerate(imgs):
        assert np.array_equal(_forward(a, [0, len(a)], geom, out)[0], E[b]), b

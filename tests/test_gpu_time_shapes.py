"""The on-chip time kernel at the limits of its CTA sizes (32 to 512 threads by
emitter count and detector size) and of its repair of the previous pixel's order:
every pixel's sorted order, by digest, and its intensity against the oracle.

The intensity bound is the one that the time path has everywhere (1e-10): the
kernel regroups an FP64 sum of n positive terms per pixel, whose rounding is of
order n 2^-53, 2e-12 at 20,480 terms."""

import numpy as np
import pytest
import torch

import oracle
from idi_b200.simulation import _core
from tests.helpers import K64, atoms, rng, sphere

pytestmark = pytest.mark.gpu


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# (emitters, detector, fwhm of the emission times): detectors of 2 x 148 x (CTAs per SM)
# pixels and more, which give each CTA size its emitter range, and of fewer; runs of 2
# and 8 positions; odd counts; narrow emission times, which move emitters by many
# places from one pixel to the next (streams, windows and warm starts given up)
CASES = [(1, 3, 5.0), (2, 70, 5.0), (65, 70, 5.0), (223, 70, 5.0), (224, 70, 5.0), (225, 69, 5.0), (1087, 70, 5.0),
         (1089, 70, 5.0), (1201, 30, 5.0), (2431, 49, 5.0), (2433, 49, 5.0), (2500, 49, 0.02), (5119, 35, 5.0),
         (5121, 35, 5.0), (6399, 30, 0.2), (6401, 30, 5.0), (10239, 25, 5.0), (10241, 25, 5.0), (20479, 13, 5.0),
         (20480, 13, 1.0)]


@pytest.mark.parametrize("n,nd,fwhm", CASES)
@pytest.mark.parametrize("settings", ["", "nf scale"])
def test_time_cta_sizes(n, nd, fwhm, settings):
    g0 = rng(1000 + n)
    at = atoms(sphere(g0, n, 0.01), g0.uniform(0, 2 * np.pi, n))
    times = g0.normal(0, fwhm / 2.35, n)
    flags, _, _ = _core.parse_settings(settings)
    geom = _core.make_geom([nd, nd + 1], 75.0, 1e5, K64, (0.0, 0.02), (0, 0), flags)
    og = oracle.geometry([nd, nd + 1], 75.0, 1e5, K64, (0.0, 0.02))
    img, dig = _core.time_forward(_gpu(at), _gpu(times), geom, 0.3, 2.0, digest=True)
    plain = _core.time_forward(_gpu(at), _gpu(times), geom, 0.3, 2.0)
    ref, ref_dig, ties = oracle.time_image_digest(og, oracle.flags_from_settings(settings), at, times, 0.3, 2.0)
    assert np.array_equal(dig.cpu().numpy().view(np.uint64), ref_dig)
    img = img.cpu().numpy()
    assert np.max(np.abs(img - ref) / np.abs(ref)) < 1e-10
    assert np.array_equal(plain.cpu().numpy(), img)


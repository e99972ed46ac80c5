"""The node rule of the band-limited evaluation (csrc/nodes.cuh) for objects of next to no phase
and for needles along the beam: the near field's exact phase and amplitude 1/|d - r|, along
one axis in extended precision."""

import numpy as np
import pytest

from helpers import rng

ld = np.longdouble


def count(phi, curve, t, fine):
    n = (max(phi + 5.0 + 9.6 * np.cbrt(phi) + 30.0 * t, 2 * (curve + 5.0 + 9.6 * np.cbrt(curve)),
             1.0 + 35.0 / np.arcsinh(0.75 / t)) if fine else
         max(phi + 3.7 + 6.33 * np.cbrt(phi) + 14.0 * t, 20.0 / np.arcsinh(1.0 / t)))
    return (int(np.ceil(n)) + 1) // 2 * 2


@pytest.mark.parametrize("fine,reach", [(True, 0.25), (True, 0.05), (True, 1e-3), (False, 3e-4)])
@pytest.mark.parametrize("t", [0.005, 0.05, 0.2, 0.4, 0.6])
@pytest.mark.parametrize("phi", [1e-4, 0.01, 0.1, 0.4, 2.0, 30.0])
def test_amplitude_interpolation(fine, reach, t, phi):
    """Relative to 1/D: within 5e-15 (FP64) and 1e-8 (split precision; 3e-4: the largest reach with
    the 1/r factor)."""
    g = rng(int(1000 * t) + int(1e4 * phi))
    half, N = ld(t), 61
    pi = ld(np.pi) + ld(1.2246467991473532e-16)
    r_max = ld(reach)
    k = ld(phi) / (half * r_max)
    for trial in range(12):
        r = g.normal(size=3) * [(1, 1, 1), (1, 0.01, 0.01), (0.01, 0.01, 1)][trial % 3]
        r = (r / np.linalg.norm(r)).astype(ld) * r_max
        u0, v0 = (ld(0), ld(0)) if trial < 6 else (ld(0.2), ld(0.1))
        e = min(reach, abs(float(r[0])) + min(1.0, float(u0 + half)) * reach) + 2 * reach ** 2
        n = count(float(k * half) * e, 0.25 * phi * t, t, fine)
        th = (2 * np.arange(n) + 1).astype(ld) * pi / (2 * n)
        x = (2 * np.arange(N) - (N - 1)).astype(ld) / (N - 1)
        d = x[:, None] - np.cos(th)
        c = np.where(np.arange(n) % 2, -1, 1) * np.sin(th) / np.where(np.abs(d) < 1e-30, ld(1e-30), d)
        L = c / c.sum(1, keepdims=True)

        def parts(u):
            p = np.stack([u + u0, np.full_like(u, v0), np.full_like(u, ld(1))], -1)
            D, dist = np.sqrt((p * p).sum(1)), np.sqrt(((p - r) ** 2).sum(1))
            ph = k * ((r @ r - 2 * (p @ r)) / (dist + D) + r[2])
            return np.stack([np.cos(ph) / dist, np.sin(ph) / dist])

        err = float(np.abs(parts(half * x) - parts(half * np.cos(th)) @ L.T).max())
        assert err < (5e-15 if fine else 1e-8), (trial, n, err)

"""The node rule of the band-limited evaluation (csrc/nodes.cuh): Chebyshev
interpolation of an emitter's field over a detector, from as many nodes as the
rule gives for the emitter's extent, stays within 1e-8 of the field.

The emitters tested sit at the image's largest distance from the origin, so this
bounds every emitter of an image; pixels are the detector's own, corners included."""

import numpy as np
import pytest

from helpers import rng

K = 2 * np.pi / (1.24 / 6400.0)


def node_count(phi, t):
    n = int(np.ceil(phi + 3.7 + 6.33 * np.cbrt(phi) + 14.0 * t))
    return (n + 1) // 2 * 2


def nodes(n):
    return np.cos((2 * np.arange(n) + 1) * np.pi / (2 * n))


def weights(n, N):
    x = (2 * np.arange(N) - (N - 1)) / max(N - 1, 1)
    d = x[:, None] - nodes(n)
    d[np.abs(d) < 1e-30] = 1e-30
    w = (-1.0) ** np.arange(n) * np.sin((2 * np.arange(n) + 1) * np.pi / (2 * n))
    c = w / d
    return c / c.sum(1, keepdims=True)


def field(u, v, D, r, near):
    """exp(i phi) at the points (u, v, D), without the pixel constant."""
    d = np.stack(np.broadcast_arrays(u, v, D), -1)
    dn = np.sqrt((d ** 2).sum(-1))
    s = d @ r / dn
    ph = K * (r[2] - s)
    if near:
        ph = ph + K / (2 * dn) * (r @ r - s * s)
    return np.exp(1j * ph)


@pytest.mark.parametrize("t", [0.01, 0.1, 0.2, 0.4, 0.6])
@pytest.mark.parametrize("phi", [0.1, 1.0, 6.0, 30.0, 120.0])
@pytest.mark.parametrize("near", [False, True])
def test_interpolation_error(t, phi, near):
    g = rng(int(1000 * t) + int(10 * phi))
    D, N = 1e5, 96
    half = t * D
    pix = np.linspace(-half, half, N)
    r_max = phi * D / (K * half)
    for trial in range(6):
        r = g.normal(size=3)
        # directions in the detector plane, along the beam and in between
        r *= [(1, 1, 1), (1, 1, 0), (0.01, 0.01, 1)][trial % 3]
        r *= r_max / np.linalg.norm(r)
        off = np.array([0.0, 0.0]) if trial < 3 else g.uniform(-0.3, 0.3, 2) * D
        rr = np.linalg.norm(r)
        n = []
        for a in (0, 1):
            s = min(1.0, (np.abs(off[a]) + half) / D)
            e = min(rr, abs(r[a]) + s * rr) * (1 + 2 * rr / D)
            n.append(node_count(K * half / D * e, t))
        vals = [half * nodes(m) + o for m, o in zip(n, off)]
        V = field(vals[0][:, None], vals[1][None, :], D, r, near)
        E = weights(n[0], N) @ V @ weights(n[1], N).T
        ref = field((pix + off[0])[:, None], (pix + off[1])[None, :], D, r, near)
        assert np.abs(E - ref).max() < 1e-8, (trial, n, np.abs(E - ref).max())


def test_sine_and_cosine_polynomials():
    """The node kernel's polynomials, in FP32, over their range."""
    x = np.linspace(-0.52, 0.52, 400001).astype(np.float32)
    f = np.float32
    z = x * x

    def horner(cs):
        p = np.full_like(z, f(cs[0]))
        for c in cs[1:]:
            p = (p.astype(np.float64) * z + c).astype(np.float32)  # one rounding, as the FMA
        return p

    sn = horner([0.07687149941921234, -0.5978690981864929, 2.5500025749206543, -5.167705059051514,
                 3.141592502593994]) * x
    cs = horner([-0.024310700595378876, 0.23489117622375488, -1.3352038860321045, 4.058708667755127,
                 -4.934802055358887, 1.0])
    # fit 6e-9, then the rounding of values up to 1 (6e-8 a step) through a degree-5 Horner
    # chain whose last two steps weigh most
    assert np.abs(sn - np.sin(np.pi * x.astype(np.float64))).max() < 2e-7
    assert np.abs(cs - np.cos(np.pi * x.astype(np.float64))).max() < 2e-7


@pytest.mark.parametrize("t", [0.02, 0.2, 0.6])
@pytest.mark.parametrize("phi", [0.1, 4.0, 30.0, 120.0])
def test_fine_grid_interpolation_error(t, phi):
    """The FP64 kernel's grid, along one axis in extended precision: within 5e-15."""
    ld = np.longdouble
    g = rng(int(100 * t) + int(phi))
    D, k, N = ld(1e5), ld(32000), 61
    half = ld(t) * D
    r_max = ld(phi) * D / (k * half)
    n = int(np.ceil(phi + 5.0 + 9.6 * np.cbrt(phi) + 30.0 * t))
    n = (n + 1) // 2 * 2
    pi = ld(np.pi) + ld(1.2246467991473532e-16)
    th = (2 * np.arange(n) + 1).astype(ld) * pi / (2 * n)
    x = (2 * np.arange(N) - (N - 1)).astype(ld) / (N - 1)
    d = x[:, None] - np.cos(th)
    c = np.where(np.arange(n) % 2, -1, 1) * np.sin(th) / np.where(np.abs(d) < 1e-30, ld(1e-30), d)
    L = c / c.sum(1, keepdims=True)
    for trial in range(9):
        r = g.normal(size=3) * [(1, 1, 1), (1, 0.01, 0.01), (0.01, 0.01, 1)][trial % 3]
        r = (r / np.linalg.norm(r)).astype(ld) * r_max
        u0, v0 = (ld(0), ld(0)) if trial < 6 else (ld(0.2) * D, ld(0.1) * D)

        def parts(u):
            p = np.stack([u + u0, np.full_like(u, v0), np.full_like(u, D)], -1)
            ph = k * (r[2] - (p * r).sum(1) / np.sqrt((p * p).sum(1)))
            return np.stack([np.cos(ph), np.sin(ph)])

        assert np.abs(parts(half * x) - parts(half * np.cos(th)) @ L.T).max() < 5e-15

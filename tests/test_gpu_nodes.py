"""Band-limited evaluation (nodes and interpolation) of the split forward: against
the cancellation-free FP64 oracle at the edges of its tiles and of its dispatch."""

from functools import partial

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from helpers import K64, atoms, rng, sphere  # noqa: E402
from idi_b200 import _native as nat  # noqa: E402
from idi_b200.simulation import _core  # noqa: E402

# 2-norm of the field error over that of the field.  Per pair, in radians (rms): the FP32
# angle in half turns 5e-8, the polynomials 3e-8 each, FP32 directions and near-field
# term 5e-8; FP32 sums over 16 emitters 8.5e-8; interpolation below 1e-8.  In quadrature
# 1.2e-7; the bound leaves a factor 2 for the pixels' uneven weights.
FIELD_2NORM = 2.4e-7
# Complex128 fields take the sums in FP64: turns in 2^-32, 4e-10 rms; polynomials 1.4e-9 at
# most; interpolation below 1e-8.
FINE_2NORM = 1.5e-8


def _err(E, ref):
    return np.linalg.norm(E - ref) / np.linalg.norm(ref)


def _forward(at, off, geom, amps=None, out=nat.OUT_C128, config=None):
    t = torch.from_numpy(np.ascontiguousarray(at)).cuda()
    a = None if amps is None else torch.from_numpy(np.ascontiguousarray(amps)).cuda()
    E = _core.forward(t, off, geom, nat.SPLIT, out, amplitudes=a, config=config).cpu().numpy()
    _core.workspace_error()
    return E, _core.evaluated_pairs()


@pytest.mark.parametrize("ndet,n,r,tilt", [
    ([64, 64], 2048, 0.01, (0, 0)),        # the smallest images that take nodes; whole tiles
    ([65, 131], 1029, 0.008, (0.1, -0.05)),  # one past a tile in both directions, ragged emitters
    ([300, 77], 517, 0.012, (0, 0.2)),
    ([1000, 24], 400, 0.006, (0, 0)),      # a strip: few nodes across
])
@pytest.mark.parametrize("settings", ["", "nf", "nf scale", "scale", "secondorder"])
def test_forward_nodes_vs_oracle(ndet, n, r, tilt, settings):
    g = rng(ndet[0] + n)
    at = atoms(sphere(g, n, r), g.uniform(0, 2 * np.pi, n))
    amp = g.uniform(0.5, 1.5, n)
    flags, _, _ = _core.parse_settings(settings)
    off = (300.0, -200.0)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, tilt, off, flags)
    oflags = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(oracle.geometry(ndet, 75.0, 1e5, K64, tilt, off), oflags, at, amp)
    for dt in (np.float32, np.float64):
        E, pairs = _forward(at, [0, n], geom, amp.astype(dt), out=nat.OUT_C64)
        assert 0 < pairs < n * ndet[0] * ndet[1] / 4
        # float32 amplitudes are the kernel's own precision: compare with theirs
        assert _err(E[0], ref) < FIELD_2NORM + 4e-8, (dt, _err(E[0], ref))


@pytest.mark.parametrize("ndet,n,r,tilt", [
    ([64, 125], 4000, 0.01, (0, 0)),       # the smallest images that take nodes for complex128
    ([65, 131], 4021, 0.008, (0.1, -0.05)),
    ([300, 77], 1400, 0.012, (0, 0.2)),
    ([1000, 24], 1391, 0.006, (0, 0)),
])
@pytest.mark.parametrize("settings", ["", "nf", "nf scale", "scale", "secondorder"])
def test_forward_nodes_fp64_sums(ndet, n, r, tilt, settings):
    g = rng(ndet[0] + n)
    at = atoms(sphere(g, n, r), g.uniform(0, 2 * np.pi, n))
    amp = g.uniform(0.5, 1.5, n).astype(np.float32)
    flags, _, _ = _core.parse_settings(settings)
    off = (300.0, -200.0)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, tilt, off, flags)
    oflags = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(oracle.geometry(ndet, 75.0, 1e5, K64, tilt, off), oflags, at, amp.astype(np.float64))
    E, pairs = _forward(at, [0, n], geom, amp)
    assert 0 < pairs < n * ndet[0] * ndet[1] / 4
    E0 = E[0]
    if "nf" in settings:  # moduli: the pixels' constant phases reach 2e8 rad, whose FP64 rounding is 2e-8
        E0, ref = np.abs(E0), np.abs(ref)
    # (the near field's 1/r factors are FP32, 6e-8 of the amplitude each)
    assert _err(E0, ref) < FINE_2NORM + (6e-8 if settings == "nf scale" else 0), _err(E0, ref)
    fewer = 31999999 // (ndet[0] * ndet[1])
    _, pairs = _forward(at[:fewer], [0, fewer], geom, amp[:fewer])
    assert pairs in (0, fewer * ndet[0] * ndet[1])


def test_mixed_batch_is_the_same_image_by_image():
    """Images on nodes, direct ones, empty ones in one batch: each the same, bit for bit, as
    alone (the fixed-point sums do not depend on how the work is cut), in fields and intensities."""
    g = rng(4)
    spec = [(4000, 0.01), (0, 0.01), (500, 0.4), (3500, 0.02), (1700, 0.01), (700, 0.01), (20001, 0.004)]
    imgs = [atoms(sphere(g, n, r), g.uniform(0, 2 * np.pi, n)) for n, r in spec]
    off = np.concatenate([[0], np.cumsum([n for n, _ in spec])])
    geom = _core.make_geom([96, 101], 75.0, 1e5, K64, flags=nat.NF)
    for out in (nat.OUT_C128, nat.OUT_I32):
        E, pairs = _forward(np.concatenate(imgs), off, geom, out=out)
        assert pairs < off[-1] * 96 * 101
        for b, a in enumerate(imgs):
            if len(a) == 0:
                assert np.all(E[b] == 0)
            elif spec[b] != (500, 0.4):  # (a small direct image alone is split over emitters)
                assert np.array_equal(E[b], _forward(a, [0, len(a)], geom, out=out)[0][0]), b


def test_more_images_than_a_group_of_node_buffers():
    """Images beyond one group's buffers (512 MB) go through the same buffers again."""
    g = rng(5)
    n, nimg = 400, 60
    pos = sphere(g, n, 0.01)
    imgs = [atoms(pos, g.uniform(0, 2 * np.pi, n)) for _ in range(nimg)]
    geom = _core.make_geom([600, 700], 75.0, 1e5, K64)
    E, pairs = _forward(np.concatenate(imgs), np.arange(nimg + 1) * n, geom, out=nat.OUT_C64)
    assert pairs < nimg * n * 600 * 700 / 4
    for b in (0, 31, 59):
        ref = oracle.wavefield(oracle.geometry([600, 700], 75.0, 1e5, K64), 0, imgs[b])
        assert _err(E[b], ref) < FIELD_2NORM + 4e-8, b  # (complex64 output)


def test_dispatch_limits():
    """What leaves the node path: an amplitude without a fixed-point sum, a detector too
    wide for its distance, too few pairs, pixel_groups = -1; the results are the direct kernels'."""
    g = rng(6)
    n = 3000
    at = atoms(sphere(g, n, 0.01), g.uniform(0, 2 * np.pi, n))
    geom = _core.make_geom([72, 64], 75.0, 1e5, K64, flags=nat.NF)
    _forward = partial(globals()["_forward"], out=nat.OUT_C64)
    full = n * 72 * 64
    E, pairs = _forward(at, [0, n], geom, np.ones(n))
    assert 0 < pairs < full / 4
    D, pairs = _forward(at, [0, n], geom, np.ones(n), config={"pixel_groups": -1})
    assert _err(E[0], D[0]) < 1e-6  # the direct kernels' 2.7e-7 and this path's
    amp = np.ones(n, np.float32)
    amp[7] = np.inf
    X, pairs = _forward(at, [0, n], geom, amp)
    assert pairs == full and not np.isfinite(X).any()
    # large and small amplitudes scale through; beyond FP32's exponents for the sums' unit
    # (2^-40, 2^100) the direct kernels take them
    for s, nodes in ((1e30, True), (1e-12, True), (1e-30, False), (1e35, False)):
        X, pairs = _forward(at, [0, n], geom, np.full(n, s, np.float32))
        assert (pairs < full / 4) == nodes and _err(X[0] / s, E[0]) < 1e-6, s
    Z, _ = _forward(at, [0, n], geom, np.zeros(n))
    assert np.all(Z == 0)
    wide = _core.make_geom([72, 64], 75.0 * 30, 1e5, K64, flags=nat.NF)  # half-extent 0.8 of the distance
    at2 = atoms(sphere(g, n, 0.0005), g.uniform(0, 2 * np.pi, n))
    W, pairs = _forward(at2, [0, n], wide)
    assert pairs in (0, full)
    ref = oracle.wavefield(oracle.geometry([72, 64], 75.0 * 30, 1e5, K64), oracle.NF | oracle.ACCURATE, at2)
    assert _err(W[0], ref) < 1e-6


@pytest.mark.parametrize("ndet,n,r,tilt", [
    ([64, 64], 600, 0.01, (0, 0)),
    ([65, 131], 1029, 0.008, (0.1, -0.05)),
    ([300, 77], 517, 0.012, (0, 0.2)),
])
@pytest.mark.parametrize("settings", ["double", "double scale", "double secondorder", "nf accurate", "nf scale accurate"])
def test_fp64_nodes_vs_oracle(ndet, n, r, tilt, settings):
    """FP64 on nodes (far field, and the near field without cancellation) against the oracle; the
    plain near field keeps the direct kernel."""
    g = rng(ndet[1] + n)
    at = atoms(sphere(g, n, r), g.uniform(0, 2 * np.pi, n))
    amp = g.uniform(0.5, 1.5, n)
    flags, prec, _ = _core.parse_settings(settings)
    assert prec == nat.DOUBLE
    t, a = torch.from_numpy(at).cuda(), torch.from_numpy(amp).cuda()
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, tilt, flags=flags)
    E = _core.forward(t, [0, n], geom, nat.DOUBLE, nat.OUT_C128, amplitudes=a).cpu().numpy()[0]
    _core.workspace_error()
    assert 0 < _core.evaluated_pairs() < n * ndet[0] * ndet[1] / 2
    of = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(oracle.geometry(ndet, 75.0, 1e5, K64, tilt), of, at, amp)
    if "nf" in settings:
        # k (|d| - d_z), up to 1e7 rad, rounds differently in the two: compare what it cancels from
        E, ref = np.abs(E), np.abs(ref)
    # phases of up to 70 rad formed in about five roundings of 2^-53 of that, on both sides
    # (1e-14 each); FP64 sums and interpolation a few 1e-16; the grid 2e-15 per emitter
    assert _err(E, ref) < 3e-14, _err(E, ref)
    one = _core.make_geom(ndet, 75.0, 1e5, K64, tilt, flags=nat.NF)
    _core.forward(t, [0, n], one, nat.DOUBLE, nat.OUT_C128, amplitudes=a)
    assert _core.evaluated_pairs() == 0


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_fp64_phase_not_finite(bad):
    """An emitter whose phase is not finite makes its FP64 image NaN, and no other image."""
    g = rng(11)
    n = 1200
    at = atoms(sphere(g, 2 * n, 0.01), g.uniform(0, 2 * np.pi, 2 * n))
    at[n + 77, 3] = bad
    geom = _core.make_geom([64, 64], 75.0, 1e5, K64)
    E = _core.forward(torch.from_numpy(at).cuda(), [0, n, 2 * n], geom, nat.DOUBLE, nat.OUT_C128).cpu().numpy()
    assert _core.evaluated_pairs() > 0
    assert np.isfinite(E[0]).all()
    assert np.isnan(E[1].real).all() and np.isnan(E[1].imag).all()


# 2-norm of the gradients' errors.  The adjoint pairs carry the forward's 1.2e-7, their FP32
# sums over at most 512 nodes 2.4e-8 sqrt(512 / 2) = 3.8e-7, and G = 4 (I - T) conj(E) about
# three times the field's relative error; 7e-7 in quadrature, times 4 for what cancels in
# the gradients of a sum of random signs.
ADJOINT_2NORM = 3e-6


def _exact_nf(ndet, tilt, off, scale, at, amp, target=None):
    """Near-field E, or with a target the gradients (position, phase, amplitude) of
    sum (|E|^2 - target)^2, in FP64 from the path difference without cancellation (the
    oracle's adjoint follows the reference's |d - r| - d_z, about 5e-7 rad a pair)."""
    M = _core.rotation(tilt[0], tilt[1], 0.0)
    x = (np.arange(ndet[0]) - ndet[0] / 2) * 75.0 + off[0]
    y = (np.arange(ndet[1]) - ndet[1] / 2) * 75.0 + off[1]
    d = np.stack([*(a.ravel() for a in np.meshgrid(x, y, indexing="ij")), np.full(x.size * y.size, 1e5)], 1) @ M.T
    r, psi = at[:, :3], at[:, 3]
    E = np.empty(len(d), complex)
    gp, gpsi, ga = np.zeros_like(r), np.zeros(len(r)), np.zeros(len(r))
    for grad in (False, True):
        if grad and target is None:
            break
        for s in range(0, len(d), 512):
            dd = d[s:s + 512]
            D = np.sqrt((dd ** 2).sum(1))[:, None]
            num = (r * r).sum(1)[None] - 2 * dd @ r.T
            L = np.sqrt(D * D + num)
            c = (dd[:, :2] ** 2).sum(1)[:, None] / (D + dd[:, 2:])
            ph = K64 * (num / (L + D) + r[:, 2][None] + c) + psi[None]
            w = 1 / L if scale else np.ones_like(L)
            e = np.exp(1j * ph)
            if not grad:
                E[s:s + 512] = (w * e) @ amp
                continue
            G = (4 * (np.abs(E[s:s + 512]) ** 2 - target.ravel()[s:s + 512]) * E[s:s + 512].conj())[:, None]
            z = G * e
            ga += (w * z.real).sum(0)
            dphi = -amp * w * z.imag
            gpsi += dphi.sum(0)
            diff = dd[:, None, :] - r[None]
            gp += np.einsum("pj,pjk->jk", -K64 * dphi / L, diff)
            gp[:, 2] += K64 * dphi.sum(0)
            if scale:
                gp += np.einsum("pj,pjk->jk", amp * z.real * w ** 3, diff)
    return E.reshape(ndet) if target is None else (gp, gpsi, ga)


@pytest.mark.parametrize("ndet,n,r,tilt", [
    ([64, 125], 4000, 0.01, (0, 0)),  # the smallest images that take nodes in differentiation
    ([65, 131], 4021, 0.008, (0.1, -0.05)),
    ([300, 77], 1400, 0.012, (0, 0.2)),
])
@pytest.mark.parametrize("settings", ["", "nf", "nf scale", "scale", "secondorder"])
def test_adjoint_nodes_vs_oracle(ndet, n, r, tilt, settings):
    """The adjoint over nodes, in a batch with a direct and an empty image, against the oracle."""
    g = rng(ndet[0] + n)
    pos, ph, amp = sphere(g, n, r), g.uniform(0, 2 * np.pi, n), g.uniform(0.5, 1.5, n)
    small = 70
    pos2, ph2 = sphere(g, small, 0.3), g.uniform(0, 2 * np.pi, small)
    flags, _, _ = _core.parse_settings(settings)
    off = (300.0, -200.0)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, tilt, off, flags)
    og = oracle.geometry(ndet, 75.0, 1e5, K64, tilt, off)
    of = oracle.flags_from_settings(settings)
    at = np.concatenate([atoms(pos, ph), atoms(pos2, ph2)])
    a = np.concatenate([amp, np.ones(small)])
    offs = [0, n, n, n + small]
    t_at, t_a = torch.from_numpy(at).cuda(), torch.from_numpy(a).cuda()
    E = _core.forward(t_at, offs, geom, nat.SPLIT, nat.OUT_C128, amplitudes=t_a)
    moved = atoms(pos + g.normal(0, 5e-5, pos.shape), ph)
    near = "nf" in settings
    field = _exact_nf(ndet, tilt, off, "scale" in settings, moved, amp) if near else oracle.wavefield(og, of, moved, amp)
    target = np.abs(field) ** 2
    gI = 2 * (E.real ** 2 + E.imag ** 2 - torch.from_numpy(target).cuda()[None])
    res = []
    for cfg in (None, {"pixel_groups": -1}):
        ga, gamp = _core.backward(t_at, offs, geom, E, gI.contiguous(), amplitudes=t_a, config=cfg)
        _core.backward_workspace_error()
        res.append((ga.cpu().numpy(), gamp.cpu().numpy()))
    (ga, gamp), (da, damp) = res
    assert not np.array_equal(ga[:n], da[:n])  # the node path was taken
    if near:
        gpos_o, gpsi_o, gamp_o = _exact_nf(ndet, tilt, off, "scale" in settings, at[:n], amp, target)
    else:
        E_o = oracle.wavefield(og, of, at[:n], amp)
        _, gpos_o, gpsi_o, gamp_o = oracle.adjoint(og, of, at[:n], amp, E_o, target)
    assert _err(ga[:n, :3], gpos_o) < ADJOINT_2NORM, _err(ga[:n, :3], gpos_o)
    assert _err(ga[:n, 3], gpsi_o) < ADJOINT_2NORM, _err(ga[:n, 3], gpsi_o)
    assert _err(gamp[:n], gamp_o) < ADJOINT_2NORM, _err(gamp[:n], gamp_o)
    assert _err(ga[n:], da[n:]) < 1e-5 and _err(gamp[n:], damp[n:]) < 1e-5  # the direct image: runs against pairs


def test_adjoint_nodes_groups_and_large_counts():
    """Images of a batch give the gradients they give alone, more of them than a group's buffers
    hold, and chunks grow where an image has many emitter blocks."""
    g = rng(12)
    counts = [300, 40000] + [300] * 30
    imgs = [atoms(sphere(g, c, 0.01), g.uniform(0, 2 * np.pi, c)) for c in counts]
    at = torch.from_numpy(np.concatenate(imgs)).cuda()
    offs = np.concatenate([[0], np.cumsum(counts)])
    geom = _core.make_geom([600, 700], 75.0, 1e5, K64, flags=nat.NF)
    E = _core.forward(at, offs, geom, nat.SPLIT, nat.OUT_C128)
    gI = (E.real ** 2 + E.imag ** 2).contiguous()
    ga, gamp = _core.backward(at, offs, geom, E, gI)
    for b in (0, 1, 31):
        lo, hi = offs[b], offs[b + 1]
        one, one_amp = _core.backward(at[lo:hi].contiguous(), [0, hi - lo], geom, E[b:b + 1].contiguous(),
                                      gI[b:b + 1].contiguous())
        assert torch.equal(ga[lo:hi], one) and torch.equal(gamp[lo:hi], one_amp), b
        da, _ = _core.backward(at[lo:hi].contiguous(), [0, hi - lo], geom, E[b:b + 1].contiguous(),
                               gI[b:b + 1].contiguous(), config={"pixel_groups": -1})
        assert _err(one.cpu().numpy(), da.cpu().numpy()) < 1e-5, b


@pytest.mark.parametrize("ndet,n,r,flat", [
    ([64, 80], 100000, 0.15, 1.0),    # wider than the detector's sampling: cells straight to the pixels
    ([200, 333], 9001, 0.03, 1.0),    # to the image's nodes; ragged in every direction
    ([300, 500], 60000, 0.02, 0.01),  # a thin sheet (one layer of cells)
    ([128, 128], 70000, 0.08, 0.3),
])
@pytest.mark.parametrize("settings", ["", "nf", "nf scale"])
def test_forward_cells_vs_oracle(ndet, n, r, flat, settings):
    """Objects cut into cells, tilted and off the origin, beside images that are not cut."""
    g = rng(n)
    pos = sphere(g, n, r) * [1, 1, flat] + [0.01, -0.02, 0.005]
    at = atoms(pos, g.uniform(0, 2 * np.pi, n))
    small = atoms(sphere(g, 900, 0.006), g.uniform(0, 2 * np.pi, 900))
    amp = g.uniform(0.5, 1.5, n + 900).astype(np.float32)
    flags, _, _ = _core.parse_settings(settings)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, (0.1, -0.2), flags=flags)
    E, pairs = _forward(np.concatenate([small, at]), [0, 900, 900 + n], geom, amp)
    assert pairs < (n + 900) * ndet[0] * ndet[1] / 2
    og = oracle.geometry(ndet, 75.0, 1e5, K64, (0.1, -0.2))
    of = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(og, of, at, amp[900:].astype(np.float64))
    assert _err(E[1], ref) < FIELD_2NORM, _err(E[1], ref)
    alone, _ = _forward(at, [0, n], geom, amp[900:])
    assert np.array_equal(alone[0], E[1])


def test_cells_degenerate_objects():
    """All emitters at one point, on a line, and one far from the rest."""
    g = rng(77)
    n = 6000
    geom = _core.make_geom([96, 96], 75.0, 1e5, K64, flags=nat.NF)
    og = oracle.geometry([96, 96], 75.0, 1e5, K64)
    for pos in (np.zeros((n, 3)) + [0.003, 0.001, -0.002],
                np.stack([g.uniform(-0.1, 0.1, n), np.zeros(n), np.zeros(n)], 1),
                np.concatenate([sphere(g, n - 1, 0.005), [[0.09, -0.08, 0.02]]])):
        at = atoms(pos, g.uniform(0, 2 * np.pi, n))
        E, _ = _forward(at, [0, n], geom)
        assert _err(E[0], oracle.wavefield(og, oracle.NF | oracle.ACCURATE, at)) < FIELD_2NORM

"""Band-limited evaluation at its edges: batches over several launches, images beside
others, differentiation outputs of cut objects, large counts, tuning, large detectors."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
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


# Complex128 fields: turns in 2^-32, 4e-10 rms; polynomials 1.4e-9 at most, FP64 sums, for the
# emitters and for their cells' turns; interpolation below 1e-8 (twice for cells).
FINE_2NORM = 1.5e-8


@pytest.mark.parametrize("ndet,n,r,flat", [
    ([64, 80], 100000, 0.15, 1.0),    # cells straight to the pixels
    ([200, 333], 9001, 0.03, 1.0),    # to the image's nodes
    ([300, 500], 60000, 0.02, 0.01),  # one layer of cells
])
@pytest.mark.parametrize("settings", ["", "nf", "nf scale"])
def test_complex128_fields_of_cut_objects(ndet, n, r, flat, settings):
    g = rng(n)
    at = atoms(sphere(g, n, r) * [1, 1, flat] + [0.01, -0.02, 0.005], g.uniform(0, 2 * np.pi, n))
    amp = g.uniform(0.5, 1.5, n).astype(np.float32)
    flags, _, _ = _core.parse_settings(settings)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64, (0.1, -0.2), flags=flags)
    E = _forward(at, [0, n], geom, nat.OUT_C128, amplitudes=torch.from_numpy(amp).cuda())[0]
    assert _core.evaluated_pairs() < n * ndet[0] * ndet[1] / 2
    of = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(oracle.geometry(ndet, 75.0, 1e5, K64, (0.1, -0.2)), of, at, amp.astype(np.float64))
    if "nf" in settings:  # moduli: the pixels' constant phases reach 2e8 rad, whose FP64 rounding is 2e-8
        E, ref = np.abs(E), np.abs(ref)
    err = np.linalg.norm(E - ref) / np.linalg.norm(ref)
    assert err < FINE_2NORM + (6e-8 if settings == "nf scale" else 0), err  # (FP32 1/r factors)


@pytest.mark.parametrize("out", [nat.OUT_C128, nat.OUT_C64])
@pytest.mark.parametrize("n,lattice", [(2500, False), (20000, False), (50000, True)])
def test_emitters_in_phase(n, lattice, out):
    """A bright peak over dark pixels: an error shared by emitters in phase, or spread by the
    interpolation from the peak, must not reach the dark pixels.  The direct kernels are the
    measure, in the dark (below three times the field of random phases) and over all."""
    g = rng(n)
    if lattice:
        m = np.stack(np.meshgrid(*[np.arange(40)] * 3, indexing="ij"), -1).reshape(-1, 3)
        pos = np.concatenate([m + o for o in ([0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5])]) * 0.00036
        pos = pos[g.choice(len(pos), n, replace=False)] - pos.mean(0)
    else:
        pos = sphere(g, n, 0.01)
    at = atoms(pos, np.zeros(n))
    ndet = [120, 121]
    geom = _core.make_geom(ndet, 170.0, 1e5, K64)
    ref = oracle.wavefield(oracle.geometry(ndet, 170.0, 1e5, K64), 0, at)
    E = _forward(at, [0, n], geom, out)[0]
    assert 0 < _core.evaluated_pairs() < n * ndet[0] * ndet[1] / 2
    D = _forward(at, [0, n], geom, out, config={"pixel_groups": -1})[0]
    dark = np.abs(ref) < 3 * np.sqrt(n)
    assert np.abs(ref).max() > 30 * np.sqrt(n) and dark.sum() > 1000
    for part in (dark, np.ones_like(dark)):
        assert np.linalg.norm((E - ref)[part]) <= np.linalg.norm((D - ref)[part])


def _far_field_extended(at, ndet, pixelsize, detz, sel):
    """The far field at the pixels `sel`, phases and sums in extended precision."""
    ld = np.longdouble
    x = ((sel // ndet[1] - ndet[0] / 2) * pixelsize).astype(ld)
    y = ((sel % ndet[1] - ndet[1] / 2) * pixelsize).astype(ld)
    D = np.sqrt(x * x + y * y + ld(detz) ** 2)
    a, k = at.astype(ld), ld(K64)
    turn = 2 * (ld(np.pi) + ld(1.2246467991473532e-16))
    E = np.empty(len(sel), complex)
    for i in range(len(sel)):
        q = [x[i] / D[i], y[i] / D[i], -(x[i] ** 2 + y[i] ** 2) / (D[i] * (D[i] + ld(detz)))]
        ph = a[:, 3] - k * (a[:, 0] * q[0] + a[:, 1] * q[1] + a[:, 2] * q[2])
        ph = ph - turn * np.rint(ph / turn)
        p = ph.astype(np.float64)
        d = (ph - p).astype(np.float64)  # cos(p + d) = cos p - d sin p
        c, s = np.cos(p), np.sin(p)
        E[i] = complex(np.sum((c - s * d).astype(ld)), np.sum((s + c * d).astype(ld)))
    return E


@pytest.mark.parametrize("n", [2000, 100_000, 1_000_000])
def test_fp64_totals_at_large_counts(n):
    """FP64 on nodes is no further from extended precision than the direct FP64 kernel, whatever
    the number of emitters."""
    g = rng(n)
    at, ndet = _image(g, n, 0.004), [64, 65]
    sel = g.choice(ndet[0] * ndet[1], 24, replace=False)
    ref = _far_field_extended(at, ndet, 75.0, 1e5, sel)
    geom = _core.make_geom(ndet, 75.0, 1e5, K64)
    errs = []
    for config in (None, {"pixel_groups": -1}):
        E = _forward(at, [0, n], geom, nat.OUT_C128, nat.DOUBLE, config=config)[0].ravel()[sel]
        assert (0 < _core.evaluated_pairs() < n * 4160 / 4) == (config is None)
        errs.append(np.linalg.norm(E - ref) / np.linalg.norm(ref))
    assert errs[0] <= errs[1], errs


@pytest.mark.parametrize("precision,out", [(nat.SPLIT, nat.OUT_C64), (nat.DOUBLE, nat.OUT_C128)])
def test_tuning_times_the_direct_images_alone(precision, out):
    """A batch all on nodes keeps the default shape, and tuning on it does not change the shape
    that direct images of the same detector and counts run with; a batch with a direct image
    is tuned on that."""
    g = rng(23)
    n, ndet = 4000, [144, 148]
    geom = _core.make_geom(ndet, 75.0, 1e5, K64)
    wide = np.concatenate([_image(g, n, 0.8) for _ in range(8)])
    off = np.arange(9) * n
    _forward(wide, off, geom, out, precision)
    assert _core.evaluated_pairs() == 8 * n * ndet[0] * ndet[1]  # direct
    ctas = _core.cta_times().size
    dense = torch.from_numpy(np.concatenate([_image(g, n, 0.01) for _ in range(8)])).cuda()
    default = ({"threads": 256, "pixels_per_thread": 4, "emitters_per_tile": 512, "ctas_per_sm": 3, "pixel_groups": 1}
               if precision == nat.SPLIT else
               {"threads": 128, "pixels_per_thread": 2, "emitters_per_tile": 128, "ctas_per_sm": 2, "pixel_groups": 1})
    for _ in range(3):
        assert _core.tune(dense, off, geom, precision, out) == default
    _forward(wide, off, geom, out, precision)
    assert _core.cta_times().size == ctas
    mixed = torch.cat([dense[:n], torch.from_numpy(wide[:7 * n]).cuda()])
    other = _core.make_geom(ndet, 75.0, 1.01e5, K64, flags=nat.SECONDORDER)  # (a key of its own: the choice is kept)
    best = _core.tune(mixed, off, other, precision, out)
    assert best["threads"] in (128, 256) and best["pixels_per_thread"] in (1, 2, 4, 8)
    assert _core.evaluated_pairs() > 0  # (the tuner's last run is a whole call)
    E = _forward(mixed.cpu().numpy(), off, other, out, precision)
    F = _forward(mixed.cpu().numpy(), off, other, out, precision, config=best)
    assert np.array_equal(E, F)


def test_detectors_of_more_pixels_than_nodes_can_be():
    """Buffers bounded by the nodes of an axis (1024) rather than by the pixels: fields and
    gradients against the direct kernels'."""
    g = rng(24)
    n, ndet = 4500, [3000, 2900]
    at = torch.from_numpy(_image(g, n, 0.004)).cuda()
    geom = _core.make_geom(ndet, 75.0, 4e5, K64, flags=nat.NF)
    E, D = (_core.forward(at, [0, n], geom, nat.SPLIT, nat.OUT_C128, config=c) for c in (None, {"pixel_groups": -1}))
    assert float((E - D).norm() / D.norm()) < 1e-6  # the direct kernels' 2.7e-7 and this path's
    gI = (E.real ** 2 + E.imag ** 2).contiguous()
    ga, da = (_core.backward(at, [0, n], geom, E, gI, config=c)[0] for c in (None, {"pixel_groups": -1}))
    _core.backward_workspace_error()
    assert not torch.equal(ga, da) and float((ga - da).norm() / da.norm()) < 1e-5


def _far_field_gradients(at, ndet, pixelsize, detz, g_intensity):
    """E, and the gradients (atoms, amplitudes) of sum g_intensity |E|^2, by torch in FP64."""
    dev = at.device
    x = (torch.arange(ndet[0], device=dev, dtype=torch.float64) - ndet[0] / 2) * pixelsize
    y = (torch.arange(ndet[1], device=dev, dtype=torch.float64) - ndet[1] / 2) * pixelsize
    X, Y = (a.reshape(-1) for a in torch.meshgrid(x, y, indexing="ij"))
    D = torch.sqrt(X * X + Y * Y + detz * detz)
    q = K64 * torch.stack([X / D, Y / D, -(X * X + Y * Y) / (D * (D + detz))], 1)
    E = torch.empty(len(q), dtype=torch.complex128, device=dev)
    ga, gamp = torch.zeros_like(at), torch.zeros(len(at), dtype=torch.float64, device=dev)
    for grad in (False, True):
        for s in range(0, len(q), 256):
            ph = at[:, 3][None] - q[s:s + 256] @ at[:, :3].T
            e = torch.complex(torch.cos(ph), torch.sin(ph))
            if not grad:
                E[s:s + 256] = e.sum(1)
                continue
            z = (2 * g_intensity.reshape(-1)[s:s + 256] * E[s:s + 256].conj())[:, None] * e
            gamp += z.real.sum(0)
            ga[:, 3] -= z.imag.sum(0)
            ga[:, :3] += z.imag.T @ q[s:s + 256]
    return E.reshape(1, *ndet), ga, gamp


# As tests/test_gpu_nodes.py: pairs 1.2e-7, FP32 sums over at most 512 nodes 3.8e-7, G about
# three times the field's relative error; 7e-7 in quadrature, times 4 for what cancels.
ADJOINT_2NORM = 3e-6


@pytest.mark.parametrize("ndet,n,r,phases", [
    ([100, 100], 60000, 0.03, 6.28),   # five chunks of 2048 pixels, 3,700 nodes
    ([64, 64], 150000, 0.019, 6.28),    # two chunks, 2,100 nodes
    ([64, 64], 150000, 0.019, 0.0),     # in phase
    ([45, 91], 150000, 0.02, 6.28),
])
def test_adjoint_more_node_chunks_than_pixel_chunks(ndet, n, r, phases):
    """Small detectors and many emitters: a chunk has at most 512 nodes, however few chunks the
    pixels make."""
    g = rng(ndet[0])
    at = torch.from_numpy(atoms(sphere(g, n, r), g.uniform(0, 1, n) * phases)).cuda()
    geom = _core.make_geom(ndet, 75.0 * 100 / max(ndet), 1e5, K64)
    g_int = torch.from_numpy(g.normal(0, 1, [1] + ndet)).cuda()
    E, ga, gamp = _far_field_gradients(at, ndet, 75.0 * 100 / max(ndet), 1e5, g_int)
    out, out_amp = _core.backward(at, [0, n], geom, E, g_int)
    direct, _ = _core.backward(at, [0, n], geom, E, g_int, config={"pixel_groups": -1})
    _core.backward_workspace_error()
    assert not torch.equal(out, direct)  # the node path was taken
    for a, b in ((out[:, :3], ga[:, :3]), (out[:, 3], ga[:, 3]), (out_amp, gamp)):
        err = float((a - b).norm() / b.norm())
        assert err < ADJOINT_2NORM, err


def test_cta_times_add_up_over_the_groups():
    """A large image in the first group of node buffers, small ones in the next: the busy time
    is the call's, not the last group's."""
    g = rng(25)
    counts = [100_000] + [400] * 59
    at = np.concatenate([_image(g, c, 0.01) for c in counts])
    geom = _core.make_geom([600, 700], 75.0, 1e5, K64)
    _forward(at[:counts[0]], [0, counts[0]], geom, nat.OUT_C64)
    alone = _core.cta_times().astype(float)
    _forward(at, np.concatenate([[0], np.cumsum(counts)]), geom, nat.OUT_C64)
    busy = _core.cta_times().astype(float)
    assert busy.sum() > 0.8 * alone.sum() and busy.size == alone.size


@pytest.mark.parametrize("pixel,r,kr", [
    (1875.0, 2e4, 0.02),  # an object a fifth of the way to the detector
    (1875.0, 4e3, 0.02),
    (160.0, 4e3, 0.1),
    (160.0, 50.0, 0.1),
])
@pytest.mark.parametrize("settings", ["nf scale accurate", "nf accurate", "double scale"])
def test_fp64_objects_of_next_to_no_phase(pixel, r, kr, settings):
    """The grid follows the near field's amplitude 1/|d - r| where the phase asks for few nodes:
    interpolation 2e-15, FP64 sums of emitters in phase and weights a few 1e-16 each."""
    g = rng(26)
    n, ndet = 600, [64, 64]
    # at the end nearest the detector, where the amplitude is sharpest
    at = atoms(sphere(g, n, 0.01 * r) + [0, 0, 0.99 * r], g.uniform(0, 0.1, n))
    flags, prec, _ = _core.parse_settings(settings)
    geom = _core.make_geom(ndet, pixel, 1e5, kr / r, flags=flags)
    E = _forward(at, [0, n], geom, nat.OUT_C128, prec)[0]
    of = oracle.flags_from_settings(settings) | (oracle.ACCURATE if "nf" in settings else 0)
    ref = oracle.wavefield(oracle.geometry(ndet, pixel, 1e5, kr / r), of, at)
    err = np.abs(E - ref).max() / np.abs(ref).max()
    assert err < 5e-15, err


@pytest.mark.parametrize("n,r,ndet", [(10000, 0.015, [256, 256]), (20000, 0.01, [200, 201])])
def test_gradients_of_small_residuals_of_cut_objects(n, r, ndet):
    """Residuals 1e-2 of the intensities: their error is the intensities' (1.5e-9 here) a hundred times
    over, beside the adjoint's own, pairs 1.2e-7 and FP32 sums over 512 nodes 3.8e-7; 4.3e-7 in
    quadrature."""
    g = rng(n)
    pos, ph = sphere(g, n, r), g.uniform(0, 2 * np.pi, n)
    at = torch.from_numpy(atoms(pos, ph)).cuda()
    near = torch.from_numpy(atoms(pos + g.normal(0, 3e-6, pos.shape), ph)).cuda()
    pixel = 75.0 * 512 / max(ndet)
    geom = _core.make_geom(ndet, pixel, 1e5, K64)
    none = torch.zeros([1] + ndet, dtype=torch.float64, device="cuda")
    exact = _far_field_gradients(at, ndet, pixel, 1e5, none)[0].abs().square()
    target = _far_field_gradients(near, ndet, pixel, 1e5, none)[0].abs().square()
    assert float((exact - target).norm() / exact.norm()) < 2e-2
    ref = _far_field_gradients(at, ndet, pixel, 1e5, 2 * (exact - target))[1]
    E = _core.forward(at, [0, n], geom, nat.SPLIT, nat.OUT_C128)
    assert _core.evaluated_pairs() < n * ndet[0] * ndet[1] / 2
    ga, _ = _core.backward(at, [0, n], geom, E, (2 * (E.real ** 2 + E.imag ** 2 - target)).contiguous())
    _core.backward_workspace_error()
    for k in (slice(0, 3), slice(3, 4)):
        err = float((ga[:, k] - ref[:, k]).norm() / ref[:, k].norm())
        assert err < 5e-7, err

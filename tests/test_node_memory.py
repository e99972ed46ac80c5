"""Workspace that the band-limited evaluation adds to a call's, by detector (host arithmetic)."""

import ctypes
import os

import numpy as np
import pytest

from idi_b200 import _native as nat
from idi_b200 import build
from idi_b200.simulation import _core

K64 = 2 * np.pi / (1.24 / 6400.0)


@pytest.fixture(autouse=True)
def _own_binding(monkeypatch):
    """The library bound with the module's present ctypes structs, whatever was reloaded before."""
    if not os.path.exists(nat.LIB_PATH):
        build.build()
    monkeypatch.setattr(nat, "_lib", None)


def _sizes(nx, ny, counts, precision=nat.SPLIT, distance=1e12):
    """(forward, forward without nodes, adjoint) workspace bytes."""
    lib = nat.load()
    geom = _core.make_geom([nx, ny], 75.0, distance, K64)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    b = nat.Batch()
    b.n_images = len(counts)
    b.offsets = off.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    b.atoms = ctypes.c_void_p(256)  # (host arithmetic: never read)
    b.amplitudes = None
    b.amp_dtype = nat.F64
    direct = _core._config({"pixel_groups": -1})
    ref = ctypes.byref
    return (lib.idiwf_forward_workspace_size(ref(geom), ref(b), precision, None),
            lib.idiwf_forward_workspace_size(ref(geom), ref(b), precision, ref(direct)),
            lib.idiwf_backward_workspace_size(ref(geom), ref(b), None))


@pytest.mark.parametrize("nx,ny", [(512, 512), (1024, 1024), (4096, 4096), (8192, 8192), (16384, 16384), (24, 4096),
                                   (4096, 24), (1, 1 << 20), (1 << 20, 1), (3, 300001), (1, (1 << 30) - 1)])
@pytest.mark.parametrize("precision", [nat.SPLIT, nat.DOUBLE])
def test_node_buffers_are_bounded(nx, ny, precision):
    """512 MB, or the smallest output; beside them the plan, the emitters' sort and the cells'
    records (20,000 emitters: 4 MB).  The adjoint's other buffers: 176 bytes a pixel, and a
    record (a chunk's sums, 24 bytes, per 512 pixels) per emitter and image."""
    fwd, direct, adj = _sizes(nx, ny, [20000], precision)
    most = max(512 << 20, 4 * nx * ny)
    assert 0 <= fwd - direct <= most + (4 << 20)
    if precision == nat.SPLIT and nx * ny < 1 << 29:
        assert adj <= 176 * (nx * ny + 2048) + 24576 * (48 + 24 * (nx * ny // 512 + 2)) + most + (4 << 20)


def test_node_sums_are_bounded_by_the_nodes():
    """An axis has at most 1024 nodes: 16 bytes each for a forward's sums, 80 for the adjoint's
    records, whatever the detector."""
    a, b = _sizes(4096, 4096, [20000]), _sizes(8192, 8192, [20000])
    rows = 4 * 4096 * 1024 * 8 + 2 * 4096 * 64 * 8  # weights and columns, twice as many
    assert (b[0] - b[1]) - (a[0] - a[1]) <= rows + (1 << 20)


@pytest.mark.parametrize("nx,ny,n", [(64, 64, 150000), (100, 100, 60000), (45, 91, 150000), (600, 700, 40000)])
def test_partial_sums_hold_chunks_of_512_nodes(nx, ny, n):
    """The adjoint's node chunks are at most 512 nodes (their sums stay in FP32) for as many nodes
    as an image of the detector may have, 24 bytes per chunk and emitter."""
    entries = min(nx * ny // 4 + 4096, (nx // 2 + 64) // 2 * 2 * ((ny // 2 + 64) // 2 * 2))
    assert _sizes(nx, ny, [n])[2] >= 24 * n * -(-entries // 512)

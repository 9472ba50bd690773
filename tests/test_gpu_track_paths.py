"""Projectors on transaxial tracks: the paths that a plain geometry leaves out.

Every case asserts the route it takes (30 or more ring pairs per track, about
3600 warps; ``capi.track_plan`` and the context's count of launches on tracks).
The other side traces LOR by LOR: a context with a step limit beyond every
path.
"""
import numpy as np
import pytest

from fir_b200 import capi
from fir_b200.geometry import ProjSpec, ScannerSpec, VolSpec
from test_track_plan import MANY_RINGS

pytestmark = pytest.mark.gpu


def contexts(scanner, geometry=capi.FIR_GEOMETRY_REFERENCE):
    track, single = capi.Context(scanner), capi.Context(scanner)
    for c in (track, single):
        c.set_option(capi.FIR_OPT_GEOMETRY, geometry)
    single.set_option(capi.FIR_OPT_STEP_LIMIT, 1 << 20)  # beyond every path: LOR by LOR
    return track, single


def forward_both(track, single, proj, vol, x):
    nb = capi.proj_geometry(proj)["n_bins"]
    got, want = np.full(nb, -1.0, np.float32), np.zeros(nb, np.float32)
    n = track.track_launch_count
    track.forward(vol, x, proj, got)
    assert track.track_launch_count == n + 1
    single.forward(vol, x, proj, want)
    assert single.track_launch_count == 0
    return got, want


def test_more_ring_pairs_than_16_bits_number():
    """Clipped LORs of ring pairs past 65536 keep their bin."""
    scanner, proj, vol = MANY_RINGS
    track, single = contexts(scanner)
    x = np.random.default_rng(1).random(vol.shape_zyx, dtype=np.float32)
    got, want = forward_both(track, single, proj, vol, x)
    np.testing.assert_array_equal(got, want)
    assert np.count_nonzero(want) > want.size / 2

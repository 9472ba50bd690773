"""Projectors on transaxial tracks: bit-identical to tracing LOR by LOR.

A launch whose LORs share tracks (48 or more ring pairs per view and
tangential bin, about 3600 warps) lists each track's crossings once.  With a
step limit set the library traces every LOR by itself, in FIR's tie form, so
the two are compared on geometries where the shared list could go wrong:
voxels that put z planes on crossings, crystals inside the volume, paths
clipped by its ends, neighbouring segments interleaved, diagonal views whose x
and y crossings coincide, ragged warps.
"""
import numpy as np
import pytest

from fir_b200 import capi
from fir_b200.geometry import OSEMParams, ProjSpec, ScannerSpec, VolSpec

pytestmark = pytest.mark.gpu

# rings, crystals, radius, pitch, tangential bins, span, segments, volume, voxel, z offset
CASES = {
    "coincident_planes": (13, 96, 130.0, 4.0, 25, 1, 25, (40, 40, 30), (4.0, 4.0, 2.0), 0.0),
    "fractional_voxels": (13, 96, 130.0, 4.0, 26, 1, 25, (41, 37, 33), (3.2, 2.5, 2.5), 0.0),
    "crystals_inside": (12, 112, 100.0, 4.0, 40, 1, 23, (72, 72, 18), (3.0, 3.0, 3.0), 0.0),
    "clipped_a_little": (14, 96, 200.0, 4.0, 25, 1, 27, (30, 30, 18), (3.0, 3.0, 3.0), 0.5),
    "interleaved": (15, 96, 150.0, 5.0, 27, 1, 29, (50, 46, 40), (3.0, 3.0, 2.0), 0.0),
    "span_3": (16, 128, 160.0, 4.0, 31, 3, 9, (47, 51, 17), (4.0, 4.0, 4.0), 0.0),
    "one_slice_voxels": (13, 96, 130.0, 4.0, 25, 1, 25, (9, 150, 64), (20.0, 1.0, 1.0), 0.0),
}


def problem(name):
    r, n, radius, pitch, tang, span, seg, size, vox, off = CASES[name]
    vol = VolSpec.centred(size, vox, off)
    return ScannerSpec.ring(r, n, radius, pitch), ProjSpec(r, n, seg, tang, span), vol


def contexts(scanner, vol):
    track, single = capi.Context(scanner), capi.Context(scanner)
    for c in (track, single):
        if any(v != int(v) for v in vol.voxel):
            c.set_option(capi.FIR_OPT_GEOMETRY, capi.FIR_GEOMETRY_EXACT)
    single.set_option(capi.FIR_OPT_STEP_LIMIT, 1 << 20)  # beyond every path: FIR's form, LOR by LOR
    return track, single


@pytest.mark.parametrize("name", sorted(CASES))
def test_forward_bit_identical(name):
    scanner, proj, vol = problem(name)
    nb = capi.proj_geometry(proj)["n_bins"]
    x = np.random.default_rng(3).random(vol.shape_zyx, dtype=np.float32)
    track, single = contexts(scanner, vol)
    got, want = np.full(nb, -1.0, np.float32), np.zeros(nb, np.float32)
    track.forward(vol, x, proj, got)
    single.forward(vol, x, proj, want)
    np.testing.assert_array_equal(got, want)
    track.forward_exp(vol, x * np.float32(0.01), proj, got)
    single.forward_exp(vol, x * np.float32(0.01), proj, want)
    np.testing.assert_array_equal(got, want)


# float atomics: a voxel sums at most ~1e4 terms in another order, each sum
# within 2^-24 of its rounding, random in sign: about 1e2 * 6e-8 / sqrt(1e4)
# of the image's norm; 1e-6 as in the repository's other atomic comparisons
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("skip", [0, 1])
def test_backward_and_ratio(name, skip):
    scanner, proj, vol = problem(name)
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(5)
    y = rng.poisson(1.0, nb).astype(np.float32)  # 37 % of the bins are 0
    x = rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)
    track, single = contexts(scanner, vol)
    track.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, skip)
    for call in ("backward", "ratio_backprojection"):
        out = []
        for c in (track, single):
            img = np.zeros(vol.shape_zyx, np.float32)
            if call == "backward":
                c.backward(proj, y, vol, img)
            else:
                c.ratio_backprojection(proj, y, vol, x, img)
            out.append(img.astype(np.float64))
        assert np.linalg.norm(out[0] - out[1]) <= 1e-6 * np.linalg.norm(out[1])
    # the same voxels are reached
    assert np.array_equal(out[0] > 0, out[1] > 0)


@pytest.mark.parametrize("bad", [np.inf, np.nan, -np.float32(3e38)])
def test_forward_of_extreme_values(bad):
    scanner, proj, vol = problem("coincident_planes")
    nb = capi.proj_geometry(proj)["n_bins"]
    x = np.random.default_rng(4).random(vol.shape_zyx, dtype=np.float32)
    x[10:12, 17, 20:23] = bad
    track, single = contexts(scanner, vol)
    got, want = np.zeros(nb, np.float32), np.zeros(nb, np.float32)
    track.forward(vol, x, proj, got)
    single.forward(vol, x, proj, want)
    np.testing.assert_array_equal(got, want)


def test_weighted_osem_and_noncontiguous_subset():
    scanner, proj, vol = problem("coincident_planes")
    # a subset's launch is below the bound; one subset is not
    prm = OSEMParams(n_iterations=2, n_subsets=1)
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(6)
    y = rng.poisson(3.0, nb).astype(np.float32)
    m = rng.random(nb, dtype=np.float32) + np.float32(0.2)
    bias = rng.random(nb, dtype=np.float32)
    track, single = contexts(scanner, vol)
    sens = np.zeros((1,) + vol.shape_zyx, np.float32)
    single.backward(proj, m, vol, sens)
    out = []
    for c in (track, single):
        img = np.ones(vol.shape_zyx, np.float32)
        c.osem(proj, y, vol, img, sens, prm, bias=bias, mult=m)
        out.append(img.astype(np.float64))
    assert np.linalg.norm(out[0] - out[1]) <= 1e-5 * np.linalg.norm(out[1])


@pytest.mark.parametrize("skip", [0, 1])
def test_batch_on_tracks(skip):
    """Problems on tracks beside one LOR by LOR (4 rings), against fir_osem."""
    names = ["coincident_planes", "span_3", "interleaved"]
    parts = [problem(n) for n in names]
    parts.append((ScannerSpec.ring(4, 64, 120.0, 4.0), ProjSpec(4, 64, 7, 21), VolSpec.centred((32, 32, 8), (4.0, 4.0, 4.0))))
    rng = np.random.default_rng(8)
    prms = [OSEMParams(n_iterations=2, n_subsets=s, convolution_interval=f, fwhm_xyz=[5.0, 5.0, 5.0], cut_radius=cut)
            for s, f, cut in ((2, 1, 0.0), (1, 0, 70.0), (3, 2, 60.0), (4, 1, 0.0))]
    ctx = capi.Context(parts[0][0])
    ctx.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, skip)
    batch = capi.Batch(ctx, [(s, p, v, q) for (s, p, v), q in zip(parts, prms)])
    data = []
    for k, ((s, p, v), q) in enumerate(zip(parts, prms)):
        nb = capi.proj_geometry(p)["n_bins"]
        y = rng.poisson(1.5, nb).astype(np.float32)
        sens = np.zeros((q.n_subsets,) + v.shape_zyx, np.float32)
        c = capi.Context(s)
        c.sensitivity(p, v, sens, q.n_subsets)
        bias = rng.random(nb, dtype=np.float32) + np.float32(0.1) if k != 1 else None
        batch.set_data(k, y, sens, bias)
        img = np.ones(v.shape_zyx, np.float32)
        c.osem(p, y, v, img, sens, q, bias=bias)
        data.append(img.astype(np.float64))
        c.close()
    for use_graph in (True, False, True):
        for k, (_, _, v) in enumerate(parts):
            batch.set_image(k, np.ones(v.shape_zyx, np.float32))
        batch.osem(use_graph=use_graph)
        for k, want in enumerate(data):
            got = batch.get_image(k).astype(np.float64)
            assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want), k
    assert batch.tune() > 0
    batch.close()
    ctx.close()

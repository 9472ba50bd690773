"""Projectors on transaxial tracks: the paths that a plain geometry leaves out.

Every case asserts the route it takes (30 or more ring pairs per track, about
3600 warps; ``capi.track_plan`` and the context's count of launches on tracks).
The other side traces LOR by LOR: a context with a step limit beyond every
path.
"""
import numpy as np
import pytest

from fir_b200 import capi
from fir_b200.geometry import OSEMParams, ProjSpec, ScannerSpec, VolSpec
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


def test_outputs_are_overwritten_and_null_is_refused():
    """Every route writes its output whole, whatever it held (the sums do not
    add to it), and refuses a missing one."""
    scanner, proj, vol = (ScannerSpec.ring(13, 96, 130.0, 4.0), ProjSpec(13, 96, 25, 25),
                          VolSpec.centred((40, 40, 30), (4.0, 4.0, 2.0)))
    assert capi.track_plan(scanner, proj, vol).osem_on_tracks
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(2)
    y = rng.poisson(1.0, nb).astype(np.float32)
    x = rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)
    track, single = contexts(scanner)
    ordered = capi.Context(scanner)
    ordered.set_option(capi.FIR_OPT_BACKPROJ_MODE, capi.FIR_BACKPROJ_DETERMINISTIC)
    floats = capi.Context(scanner)
    floats.set_option(capi.FIR_OPT_TRAVERSAL, capi.FIR_TRAVERSAL_FLOAT)
    import torch

    for c in (track, single, ordered, floats):
        for n_subsets in (1, 4):
            out = []
            for fill in (0.0, 1e6):
                b = torch.full((n_subsets,) + vol.shape_zyx, fill, device="cuda")
                s = torch.full_like(b, fill)
                r = torch.full(vol.shape_zyx, fill, device="cuda")
                dy, dx = torch.from_numpy(y).cuda(), torch.from_numpy(x).cuda()
                c.backward(proj, dy, vol, b, n_subsets)
                c.sensitivity(proj, vol, s, n_subsets)
                c.ratio_backprojection(proj, dy, vol, dx, r, n_subsets=n_subsets, subset=n_subsets - 1)
                c.synchronize()
                out.append([t.double() for t in (b, s, r)])
            for a, b in zip(*out):
                assert float((a - b).norm()) <= 1e-6 * float(a.norm())
    L, pd, vd = capi.lib(), capi.C.byref(capi.proj_desc(proj)), capi.C.byref(capi.vol_desc(vol, 1))
    refused = 1  # FIR_ERR_INVALID_ARGUMENT
    assert L.fir_sensitivity(track.handle, pd, vd, None, 1) == refused
    assert L.fir_backward(track.handle, pd, capi._ptr(y), vd, None, 1) == refused


def test_first_backprojection_may_be_captured_above_l2():
    """Above L2 the LOR-by-LOR backprojection needs no scratch, so a context's
    first call can be captured; tracks need scratch and step back."""
    import torch

    scanner, proj = ScannerSpec.ring(16, 256, 300.0, 4.0), ProjSpec(16, 256, 31, 99)
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    nz = int(l2 / 8 / (280 * 280)) + 2
    vol = VolSpec.centred((280, 280, nz), (2.0, 2.0, 2.0))
    assert capi.track_plan(scanner, proj, vol).osem_on_tracks
    nb = capi.proj_geometry(proj)["n_bins"]
    y = torch.rand(nb, device="cuda")
    out = torch.zeros(vol.shape_zyx, device="cuda")
    eager, first = capi.Context(scanner), capi.Context(scanner)
    eager.backward(proj, y, vol, out)
    eager.synchronize()
    assert eager.track_launch_count == 1
    want = out.double()
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        first.backward(proj, y, vol, out)
    assert first.track_launch_count == 0
    graph.replay()
    torch.cuda.synchronize()
    assert float((out.double() - want).norm()) <= 1e-6 * float(want.norm())
    # with its scratch the context's next calls run on tracks, captured ones too
    first.backward(proj, y, vol, out)
    assert first.track_launch_count == 1
    again = torch.cuda.CUDAGraph()
    out.zero_()
    with torch.cuda.graph(again):
        first.backward(proj, y, vol, out)
    assert first.track_launch_count == 2
    again.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert float((out.double() - want).norm()) <= 1e-6 * float(want.norm())


def test_captured_launch_keeps_its_scratch():
    """A later call on tracks leaves the scratch of a captured LOR-by-LOR
    sub-iteration in place."""
    import torch

    scanner, proj, vol = (ScannerSpec.ring(13, 96, 130.0, 4.0), ProjSpec(13, 96, 25, 25),
                          VolSpec.centred((40, 40, 30), (4.0, 4.0, 2.0)))
    assert capi.track_plan(scanner, proj, vol).osem_on_tracks
    assert not capi.track_plan(scanner, proj, vol, n_subsets=4).osem_on_tracks
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(3)
    y = torch.from_numpy(rng.poisson(2.0, nb).astype(np.float32)).cuda()
    x0 = torch.from_numpy(rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)).cuda()
    sens = torch.ones(vol.shape_zyx, device="cuda")
    prm = OSEMParams(n_subsets=4)
    ctx = capi.Context(scanner)
    x = x0.clone()
    ctx.osem_subiteration(proj, y, vol, x, sens, prm, 1, 1)
    want = x.double()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.osem_subiteration(proj, y, vol, x, sens, prm, 1, 1)
    assert ctx.track_launch_count == 0
    full = torch.empty(vol.shape_zyx, device="cuda")
    ctx.sensitivity(proj, vol, full)
    ctx.synchronize()
    assert ctx.track_launch_count == 1
    x.copy_(x0)
    graph.replay()
    torch.cuda.synchronize()
    assert float((x.double() - want).norm()) <= 1e-6 * float(want.norm())


def test_a_filtered_subiteration_leaves_the_filter_its_scratch():
    """A context whose sub-iteration filtered in one launch captures its first
    fir_convolve, as after one that filtered in passes."""
    import torch

    scanner, proj = ScannerSpec.ring(4, 64, 120.0, 4.0), ProjSpec(4, 64, 7, 21)
    vol = VolSpec.centred((32, 32, 8), (4.0, 4.0, 4.0))
    fwhm = [4.0, 4.0, 4.0]
    y = torch.ones(capi.proj_geometry(proj)["n_bins"], device="cuda")
    x = torch.rand(vol.shape_zyx, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda")
    want = x.clone()
    eager, ctx = capi.Context(scanner), capi.Context(scanner)
    eager.convolve(vol, want, fwhm)
    image = torch.ones_like(x)
    ctx.osem_subiteration(proj, y, vol, image, torch.ones_like(x), OSEMParams(convolution_interval=1, fwhm_xyz=fwhm),
                          0, 1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.convolve(vol, x, fwhm)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want)


def test_scratch_leaves_room_for_the_rest_of_the_call():
    """Where the device has room for the tracks' scratch but not for the
    filter's as well, the sub-iteration runs LOR by LOR."""
    import torch

    scanner, proj = ScannerSpec.ring(16, 192, 170.0, 4.0), ProjSpec(16, 192, 31, 71)
    vol = VolSpec.centred((256, 256, 256), (1.0, 1.0, 1.0))
    assert capi.track_plan(scanner, proj, vol).osem_on_tracks
    voxels = 256 ** 3
    y = torch.ones(capi.proj_geometry(proj)["n_bins"], device="cuda")
    sens = torch.ones(vol.shape_zyx, device="cuda")
    prm = OSEMParams(n_subsets=1, convolution_interval=1, fwhm_xyz=(4.0, 4.0, 4.0))

    def run(limit, launches_on_tracks):
        ctx = capi.Context(scanner)
        if limit:
            ctx.set_option(capi.FIR_OPT_STEP_LIMIT, 1 << 20)
        x = torch.ones(vol.shape_zyx, device="cuda")
        ctx.osem_subiteration(proj, y, vol, x, sens, prm, 0, 1)
        ctx.synchronize()
        assert ctx.track_launch_count == launches_on_tracks
        return x.cpu().double()

    run(False, 1)  # (loads the kernels)
    want = run(True, 0)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # the image takes 4 bytes per voxel, the tracks' scratch 24, the filter's 8; LOR
    # by LOR it is 8, and 8 for the filter and the backprojection
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (4 + 28) * voxels, dtype=torch.uint8, device="cuda")
    try:
        got = run(False, 0)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert float((got - want).norm()) <= 1e-6 * float(want.norm())


def test_a_batch_without_room_for_the_accumulators():
    """It runs LOR by LOR: 20 bytes per voxel, on tracks 32."""
    import torch

    scanner, proj = ScannerSpec.ring(16, 192, 170.0, 4.0), ProjSpec(16, 192, 31, 71)
    vol = VolSpec.centred((256, 256, 256), (1.0, 1.0, 1.0))
    assert capi.track_plan(scanner, proj, vol).osem_on_tracks
    y = np.random.default_rng(8).poisson(3.0, capi.proj_geometry(proj)["n_bins"]).astype(np.float32)
    ones = np.ones(vol.shape_zyx, np.float32)
    ctx = capi.Context(scanner)

    def run():
        batch = capi.Batch(ctx, [(scanner, proj, vol, OSEMParams())])
        batch.set_data(0, y, ones)
        batch.set_image(0, ones)
        batch.osem()
        out = batch.get_image(0).astype(np.float64)
        batch.close()
        return out

    want = run()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 26 * 256 ** 3, dtype=torch.uint8, device="cuda")
    try:
        got = run()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


# Sums of floats in another order: 1e-6 as in the repository's other
# comparisons of float atomics.
@pytest.mark.parametrize("occupied", [0.0, 1e-4, 0.1, 0.159, 0.161, 0.4, 0.649, 0.651, 1.0])
@pytest.mark.parametrize("span", [1, 3])
def test_skipped_bins_at_any_occupancy(occupied, span):
    """Below 65 % of the bins non-zero (backprojection: 16 %) a launch on tracks
    leaves them to the general walk, above it traces all (packs them); both equal
    the LOR-by-LOR route."""
    if span == 1:
        scanner, proj, vol = (ScannerSpec.ring(15, 96, 150.0, 5.0), ProjSpec(15, 96, 29, 27),
                              VolSpec.centred((50, 46, 40), (3.0, 3.0, 2.0)))
    else:
        scanner, proj, vol = (ScannerSpec.ring(16, 128, 160.0, 4.0), ProjSpec(16, 128, 9, 31, 3),
                              VolSpec.centred((47, 51, 17), (4.0, 4.0, 4.0)))
    assert capi.track_plan(scanner, proj, vol, skip_zero=True).osem_on_tracks
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(4)
    y = rng.poisson(3.0, nb).astype(np.float32) + np.float32(1)
    keep = int(round(occupied * nb))
    y[rng.permutation(nb)[keep:]] = 0
    m = rng.random(nb, dtype=np.float32) + np.float32(0.2)
    x = rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)
    track, single = contexts(scanner)
    track.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, 1)
    sens = np.ones((1,) + vol.shape_zyx, np.float32)
    out = []
    for c in (track, single):
        back, ratio, osem = (np.zeros(vol.shape_zyx, np.float32) for _ in range(3))
        c.backward(proj, y, vol, back)
        c.ratio_backprojection(proj, y, vol, x, ratio)
        osem[:] = x
        c.osem(proj, y, vol, osem, sens, OSEMParams(n_iterations=1, n_subsets=1), mult=m)
        out.append([a.astype(np.float64) for a in (back, ratio, osem)])
    assert track.track_launch_count == 3 and single.track_launch_count == 0
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
        assert np.array_equal(a > 0, b > 0)


# rings, crystals, segments, span, tangential bins, size, voxel, z offset, geometry, block size
REF, EXACT = capi.FIR_GEOMETRY_REFERENCE, capi.FIR_GEOMETRY_EXACT
PATHS = {
    # z clips 2 to 3 % of the LORs, at both ends of the volume or at one
    "clipped": (16, 192, 31, 1, 71, (50, 46, 28), (4.0, 4.0, 2.0), 0.0, REF, 0),
    "clipped_one_end": (16, 192, 31, 1, 71, (50, 46, 30), (4.0, 4.0, 2.0), 2.5, REF, 0),
    "clipped_blocks_of_256": (16, 192, 31, 1, 71, (50, 46, 28), (4.0, 4.0, 2.0), 0.0, REF, 256),
    "clipped_blocks_of_32": (16, 192, 31, 1, 71, (50, 46, 28), (4.0, 4.0, 2.0), 0.0, REF, 32),
    # two tracks per block
    "clipped_two_tracks": (10, 384, 19, 1, 71, (90, 90, 18), (3.0, 3.0, 2.0), 0.0, REF, 0),
    # extents truncated to whole millimetres: paths leave the slices early
    "truncated": (16, 192, 31, 1, 71, (50, 46, 27), (3.3, 3.7, 2.4), 0.0, REF, 0),
    # extents that are not whole, two plane offsets per segment
    "fractional": (16, 192, 31, 1, 71, (51, 45, 40), (3.3, 2.7, 1.6), 0.0, EXACT, 0),
    "span_3_clipped": (20, 192, 13, 3, 71, (47, 51, 37), (4.0, 4.0, 2.0), 0.0, REF, 0),
}


def path_case(name):
    r, n, seg, span, tang, size, voxel, off, geometry, block = PATHS[name]
    scanner = ScannerSpec.ring(r, n, 170.0, 4.0)
    proj, vol = ProjSpec(r, n, seg, tang, span), VolSpec.centred(size, voxel, off)
    plan = capi.track_plan(scanner, proj, vol, geometry=geometry, block_size=block)
    assert plan.forward_on_tracks and plan.backward_on_tracks and plan.osem_on_tracks
    assert (plan.general > 1e-3) == (name != "fractional")
    assert plan.block_tracks == {"clipped_two_tracks": 2, "clipped_blocks_of_256": 2}.get(name, 1)
    track, single = contexts(scanner, geometry)
    track.set_option(capi.FIR_OPT_BLOCK_SIZE, block)
    return track, single, proj, vol


@pytest.mark.parametrize("name", sorted(PATHS))
def test_projection_is_bit_identical(name):
    track, single, proj, vol = path_case(name)
    x = np.random.default_rng(5).random(vol.shape_zyx, dtype=np.float32)
    got, want = forward_both(track, single, proj, vol, x)
    np.testing.assert_array_equal(got, want)
    track.forward_exp(vol, x * np.float32(0.01), proj, got)
    single.forward_exp(vol, x * np.float32(0.01), proj, want)
    np.testing.assert_array_equal(got, want)


# A voxel sums some 1e4 floats: 1e-6 of the norm as in the repository's other
# comparisons of float atomics, here against sums in 64 bits of the same terms
# (the multi-frame backprojection, which traces LOR by LOR).
@pytest.mark.parametrize("name", sorted(PATHS))
@pytest.mark.parametrize("skip", [0, 1])
def test_backprojections_agree(name, skip):
    track, single, proj, vol = path_case(name)
    nb = capi.proj_geometry(proj)["n_bins"]
    rng = np.random.default_rng(6)
    y = rng.poisson(1.0, nb).astype(np.float32)  # 37 % of the bins are 0
    m = rng.random(nb, dtype=np.float32) + np.float32(0.2)
    bias = rng.random(nb, dtype=np.float32)
    x = rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)
    track.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, skip)
    sens = np.ones((1,) + vol.shape_zyx, np.float32)
    back, ones, ratio = (np.zeros(vol.shape_zyx, np.float32) for _ in range(3))
    track.backward(proj, y, vol, back)
    track.sensitivity(proj, vol, ones)
    track.ratio_backprojection(proj, y, vol, x, ratio, bias=bias)
    osem = x.copy()
    track.osem(proj, y, vol, osem, sens, OSEMParams(n_iterations=1, n_subsets=1), bias=bias, mult=m)
    assert track.track_launch_count == 4

    def wide(bins):
        out = np.zeros((1,) + vol.shape_zyx)
        single.backward_frames(proj, bins[None].astype(np.float64), vol, out)
        return out[0]

    def over(estimate):
        with np.errstate(divide="ignore", invalid="ignore"):
            return np.where(estimate > 1e-5, y / estimate, np.float32(0))

    line = np.zeros(nb, np.float32)
    single.forward(vol, x, proj, line)
    want_osem = wide(over(line * m + bias) * m)
    want_osem = np.where(want_osem > 1e-5, x * want_osem, 0.0)
    assert single.track_launch_count == 0
    for got, want in ((back, wide(y)), (ones, wide(np.ones(nb, np.float32))), (ratio, wide(over(line + bias))),
                      (osem, want_osem)):
        assert np.linalg.norm(got.astype(np.float64) - want) <= 1e-6 * np.linalg.norm(want)
        assert np.array_equal(got != 0, want != 0)


def test_rounding_is_no_larger_than_lor_by_lor():
    """The backprojection's distance from sums in 64 bits, on a subset of the
    clinical scanner's bins."""
    import torch

    scanner, proj = ScannerSpec.ring(32, 512, 400.0, 4.0), ProjSpec(32, 512, 63, 125)
    vol = VolSpec.centred((200, 200, 64), (3.0, 3.0, 3.0))
    assert capi.track_plan(scanner, proj, vol, n_subsets=16).backward_on_tracks
    track, single = contexts(scanner)
    gen = torch.Generator(device="cuda").manual_seed(7)
    nb = capi.proj_geometry(proj)["n_bins"]
    y = 0.5 + torch.rand(nb, generator=gen, device="cuda")
    wide = torch.zeros((1,) + vol.shape_zyx, device="cuda", dtype=torch.float64)
    at, only = 0, torch.zeros_like(y)
    for seg in range(-31, 32):  # the views of subset 3
        n = (32 - abs(seg)) * 125
        only[at:at + 256 * n].view(256, n)[3::16] = y[at:at + 256 * n].view(256, n)[3::16]
        at += 256 * n
    single.backward_frames(proj, only[None].double(), vol, wide)
    error = []
    for c in (track, single):
        out = torch.zeros((16,) + vol.shape_zyx, device="cuda")
        c.backward(proj, y, vol, out, 16)
        c.synchronize()
        error.append(float((out[3].double() - wide[0]).norm() / wide.norm()))
    assert error[0] <= error[1] <= 1e-6, error


@pytest.mark.parametrize("occupied", [0.01, 0.6])
def test_a_large_problem_of_a_batch_skips_bins(occupied):
    """Above 2^22 LORs per subset a problem has launches of its own; they pack
    the non-zero bins of their blocks too."""
    scanner, proj = ScannerSpec.ring(32, 256, 300.0, 4.0), ProjSpec(32, 256, 63, 65)
    vol = VolSpec.centred((60, 56, 64), (4.0, 4.0, 2.0))
    nb = capi.proj_geometry(proj)["n_bins"]
    assert nb >= 1 << 22 and capi.track_plan(scanner, proj, vol, skip_zero=True).osem_on_tracks
    rng = np.random.default_rng(10)
    y = np.where(rng.random(nb) < occupied, rng.integers(1, 5, nb), 0).astype(np.float32)
    ones = np.ones(vol.shape_zyx, np.float32)
    ctx, single = capi.Context(scanner), capi.Context(scanner)
    single.set_option(capi.FIR_OPT_STEP_LIMIT, 1 << 20)
    ctx.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, 1)
    batch = capi.Batch(ctx, [(scanner, proj, vol, OSEMParams())])
    batch.set_data(0, y, ones)
    batch.set_image(0, ones)
    batch.osem()
    got = batch.get_image(0).astype(np.float64)
    batch.close()
    # (sums in 64 bits, as above: LOR by LOR, float sums of this many LORs differ
    # from them by more than those on tracks)
    line, want = np.zeros(nb, np.float32), np.zeros((1,) + vol.shape_zyx)
    single.forward(vol, ones, proj, line)
    ratio = np.divide(y, line, out=np.zeros_like(y), where=line > 1e-5)
    single.backward_frames(proj, ratio[None].astype(np.float64), vol, want)
    want = np.where(want[0] > 1e-5, want[0], 0.0)
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    assert np.array_equal(got > 0, want > 0)

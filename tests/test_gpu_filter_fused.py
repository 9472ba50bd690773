"""A sub-iteration's filter in one launch equals its separate passes, bit for bit.

Volumes up to 2^20 voxels with narrow taps are filtered by one kernel (tiles of
32 x 8 x 4 voxels with the taps' halo) that also restores the edge and applies
the cut; larger ones, and wider taps, by three passes.  In the
deterministic mode a sub-iteration without filter followed by fir_convolve
and fir_cut_circle gives the same image.
"""
import numpy as np
import pytest

from fir_b200 import capi
from fir_b200.geometry import OSEMParams, ProjSpec, ScannerSpec, VolSpec

pytestmark = pytest.mark.gpu

SCANNER = ScannerSpec.ring(6, 64, 110.0, 4.0)
PROJ = ProjSpec(6, 64, 11, 21)


@pytest.mark.parametrize("size,voxel,fwhm,cut", [
    ((32, 8, 4), 4.0, (4.0, 4.0, 4.0), 0.0),     # one tile
    ((33, 9, 5), 4.0, (4.0, 4.5, 3.0), 0.0),     # one voxel past it
    ((31, 7, 3), 5.0, (5.0, 5.0, 5.0), 60.0),    # ragged, edge restored and cut
    ((31, 7, 3), 3.0, (9.0, 9.0, 9.0), 30.0),    # taps wider than the volume: three passes
    ((1, 40, 1), 4.0, (6.0, 6.0, 6.0), 0.0),     # single columns
    ((65, 63, 9), 2.0, (4.0, 6.0, 8.0), 55.0),
    ((40, 40, 12), 2.0, (20.0, 20.0, 20.0), 0.0),  # wide taps: three passes
    ((130, 128, 64), 1.0, (4.0, 4.0, 4.0), 60.0),  # above 2^20 voxels: three passes
])
def test_subiteration_filter_matches_passes(size, voxel, fwhm, cut):
    vol = VolSpec.centred(size, (voxel,) * 3)
    nb = capi.proj_geometry(PROJ)["n_bins"]
    rng = np.random.default_rng(9)
    y = rng.poisson(4.0, nb).astype(np.float32)
    x = rng.random(vol.shape_zyx, dtype=np.float32) + np.float32(0.1)
    ctx = capi.Context(SCANNER)
    ctx.set_option(capi.FIR_OPT_BACKPROJ_MODE, capi.FIR_BACKPROJ_DETERMINISTIC)
    sens = np.zeros(vol.shape_zyx, np.float32)
    ctx.sensitivity(PROJ, vol, sens, 1)
    got, want = x.copy(), x.copy()
    filtered = OSEMParams(n_subsets=1, cut_radius=cut, convolution_interval=1, fwhm_xyz=list(fwhm))
    ctx.osem_subiteration(PROJ, y, vol, got, sens, filtered, 0, 1)
    ctx.osem_subiteration(PROJ, y, vol, want, sens, OSEMParams(n_subsets=1), 0, 1)
    ctx.convolve(vol, want, fwhm, cut)
    ctx.cut_circle(vol, want, cut)
    np.testing.assert_array_equal(got, want)
    assert np.any(got != x)
    ctx.close()

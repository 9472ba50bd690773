"""CPU tests of the rule that puts projector launches on transaxial tracks, and
of the arithmetic by which a block numbers the LORs it leaves to the general
walk.  No GPU call is made."""
import subprocess

import pytest

from fir_b200 import capi
from fir_b200.build import CSRC, CXX, NVCC
from fir_b200.geometry import ProjSpec, ScannerSpec, VolSpec

# 400 rings and 255 segments: more ring pairs per track than 16 bits number;
# the volume ends inside the outermost rings
MANY_RINGS = (ScannerSpec.ring(400, 64, 200.0, 2.0), ProjSpec(400, 64, 255, 5),
              VolSpec.centred((20, 20, 75), (10.0, 10.0, 10.0)))

PLACES = r"""
#include "internal.h"
#include <cstdio>
#include <vector>
// pairs, share, tracks per block
int main()
{
  const int plans[][3] = {{85744, 256, 1}, {1023, 256, 1}, {305, 305, 1}, {30, 30, 8}, {64, 64, 4}, {100000, 1024, 1}};
  for (const auto& q : plans)
  {
    fir::ColumnPlan p{};
    p.pairs = q[0];
    p.share = q[1];
    p.per_block = q[2];
    p.blocks = (p.pairs + p.share - 1) / p.share;
    const unsigned room = (unsigned)(p.per_block * p.share);
    for (int block = 0; block < p.blocks; ++block)
    {
      std::vector<char> seen(room, 0);
      const int begin = block * p.share;
      for (int group = 0; group < p.per_block; ++group)
      {
        for (int pair = begin; pair < begin + p.share && pair < p.pairs; ++pair)
        {
          const unsigned place = fir::block_place(p, fir::BlockLor{group, pair - begin});
          if (place >= room || seen[place]++)
          {
            std::printf("pairs %d: place %u of %u\n", p.pairs, place, room);
            return 1;
          }
          const fir::BlockLor l = fir::block_lor(p, place);
          if (l.group != group || begin + l.offset != pair)
          {
            std::printf("pairs %d: pair %d of track %d came back as %d of %d\n", p.pairs, pair, group,
                        begin + l.offset, l.group);
            return 1;
          }
        }
      }
    }
  }
  return 0;
}
"""


def test_places_in_a_block_are_distinct_and_come_back(tmp_path):
    src = tmp_path / "places.cu"
    src.write_text(PLACES)
    exe = str(tmp_path / "places")
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-ccbin", CXX, "-I", CSRC, "-o", exe, str(src)],
                   check=True)
    done = subprocess.run([exe], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def test_plan_of_many_rings():
    plan = capi.track_plan(*MANY_RINGS)
    assert plan.forward_on_tracks and plan.ring_pairs == 85744 and plan.general > 0
    # a block's list of LORs for the general walk holds a place for each
    assert plan.block_tracks * plan.block_pairs * 4 <= plan.shared_bytes


def test_plan_rejects_what_the_projectors_reject():
    scanner, proj, vol = MANY_RINGS
    for bad in (dict(n_subsets=5), dict(n_subsets=2, subset=2), dict(block_size=48), dict(geometry=7)):
        with pytest.raises(capi.FirError):
            capi.track_plan(scanner, proj, vol, **bad)


def count_general(scanner, proj, vol, geometry):
    """Share of the LORs that meet the volume which a lane gives to the general
    walk: z clips them, or they leave the traversal's slices before they end.
    Every fifth view, every third tangential bin, all ring pairs."""
    import ctypes as C

    import numpy as np

    eps = 1e-5
    xy, z = np.zeros((scanner.n_crystals_per_ring, 2)), np.zeros(2 * scanner.n_rings - 1)
    a, b = C.c_int(), C.c_int()
    capi.lib().fir_scanner_tables(C.byref(capi.scanner_desc(scanner)), xy.ctypes.data, z.ctypes.data, C.byref(a),
                                  C.byref(b))
    ends = []
    for seg in range(-(proj.n_segments // 2), proj.n_segments // 2 + 1):
        for k in range(proj.n_rings - abs(seg)):
            ends.append((2 * (k + max(seg, 0)), 2 * (k + max(-seg, 0))))
    ends = np.array(ends)
    z1, z2 = z[ends[:, 0]], z[ends[:, 1]]
    vox, size = np.array(vol.voxel), np.array(vol.size)
    ext = np.trunc(vox) if geometry == capi.FIR_GEOMETRY_REFERENCE else vox
    low = np.array([vol.offset[0] - vox[0] / 2, vol.offset[1] - vox[1] / 2, vol.offset[2] - size[2] * vox[2] / 2])
    high = low + size * vox
    n, nt = scanner.n_crystals_per_ring, proj.n_tang_coords
    meeting = general = 0
    for view in range(0, n // 2, 5):
        for t in range(-(nt // 2), nt - nt // 2, 3):
            shift = t // 2 if t >= 0 else int((t - 1) / 2)
            p1, p2 = xy[(view + shift + abs(t) % 2) % n], xy[(view + n // 2 - shift) % n]
            amin, amax = 0.0, 1.0
            for d in (0, 1):
                df = p2[d] - p1[d]
                if abs(df) > eps:
                    q = sorted(((low[d] - p1[d]) / df, (high[d] - p1[d]) / df))
                    amin, amax = max(amin, q[0]), min(amax, q[1])
                elif not low[d] <= p1[d] <= high[d]:
                    amax = -1.0
            if amin >= amax:
                continue
            df = z2 - z1
            moves, up = np.abs(df) > eps, df > eps
            df = np.where(moves, df, eps)
            q1, q2 = (low[2] - z1) / df, (high[2] - z1) / df
            into, out = np.where(moves, np.minimum(q1, q2), 0), np.where(moves, np.maximum(q1, q2), 1)
            misses = ~moves & ((z1 < low[2]) | (z1 > high[2])) | (np.maximum(into, amin) >= np.minimum(out, amax))
            dz = np.abs(ext[2] / df)
            ind = np.clip(np.trunc((z1 + df * amin - low[2]) / ext[2]), 0, size[2] - 1)
            first = np.where(moves, (low[2] + ext[2] * ind - z1) / df, 1.0) + np.where(up, dz, 0)
            leaves = first + np.where(up, size[2] - 1 - ind, ind) * dz
            shared = (into <= amin) & (out >= amax) & (dz > 4 * eps) & (leaves > amax + 4 * eps)
            meeting += np.count_nonzero(~misses)
            general += np.count_nonzero(~misses & ~shared)
    return general / meeting


@pytest.mark.parametrize("rings,size,voxel,offset,geometry", [
    (17, (128, 128, 33), (3.0, 3.0, 2.0), 0.0, 0),     # covers the scanner
    (17, (128, 128, 31), (3.0, 3.0, 2.0), 0.0, 0),     # ends inside the last rings
    (17, (128, 96, 24), (3.0, 3.0, 2.0), 7.0, 0),      # off centre
    (17, (128, 128, 8), (3.0, 3.0, 2.0), 0.0, 0),      # far shorter
    (24, (160, 160, 52), (3.0, 3.0, 1.9), 0.0, 0),     # slices truncated to 1 mm
    (24, (160, 160, 52), (3.0, 3.0, 1.9), 0.0, 1),     # the same, exact
    (24, (192, 192, 40), (2.5, 2.5, 2.5), 0.0, 0),     # all extents truncated
    (8, (200, 200, 11), (3.0, 3.0, 3.0), 0.0, 0),      # crystals within the volume's corners
])
def test_share_of_general_lors(rings, size, voxel, offset, geometry):
    """The estimate samples 40 tracks: within 15 % of the count."""
    scanner, proj = ScannerSpec.ring(rings, 256, 320.0, 4.0), ProjSpec(rings, 256, 2 * rings - 1, 91)
    vol = VolSpec.centred(size, voxel, offset)
    counted = count_general(scanner, proj, vol, geometry)
    plan = capi.track_plan(scanner, proj, vol, geometry=geometry)
    assert abs(plan.general - counted) <= 0.15 * counted + 1e-4
    # where many are, the fused kernel and the projection stay LOR by LOR
    if counted > 0.1:
        assert not plan.osem_on_tracks and not plan.forward_on_tracks
    if counted == 0.0 and plan.stops <= 2.2:
        assert plan.osem_on_tracks and plan.forward_on_tracks and plan.backward_on_tracks


def test_few_rings_and_long_volumes():
    """Six rings fill half of a warp: only the backprojection gains.  A volume of
    more slices than the copies' tile grid stays LOR by LOR."""
    plan = capi.track_plan(ScannerSpec.ring(6, 384, 350.0, 4.0), ProjSpec(6, 384, 11, 125),
                           VolSpec.centred((170, 170, 20), (3.0, 3.0, 2.0)))
    assert (plan.forward_on_tracks, plan.backward_on_tracks, plan.osem_on_tracks) == (0, 1, 0)
    scanner, proj = ScannerSpec.ring(16, 192, 170.0, 4.0), ProjSpec(16, 192, 31, 71)
    for nz, on in ((65535 * 32, 1), (65535 * 32 + 1, 0)):
        plan = capi.track_plan(scanner, proj, VolSpec.centred((1, 1, nz), (2.0, 2.0, 2.0)))
        assert plan.backward_on_tracks == on and plan.osem_on_tracks == on


# rings, crystals, radius, pitch, size, voxel; routes (forward, backward, fused).
# Exact geometry, span 1, nothing clipped but where named.
@pytest.mark.parametrize("rings,crystals,radius,pitch,size,voxel,routes", [
    (16, 256, 250.0, 4.0, (64, 64, 43), (4.0, 4.0, 1.6), (1, 1, 1)),        # full warps, 1.8 stops
    (16, 256, 250.0, 4.0, (64, 64, 38), (4.0, 4.0, 1.8181818), (0, 1, 1)),  # 3.2
    (16, 256, 250.0, 4.0, (64, 64, 54), (4.0, 4.0, 1.3), (0, 1, 0)),        # 6.5
    (12, 320, 250.0, 4.0, (64, 64, 19), (4.0, 4.0, 3.0), (1, 1, 1)),        # three quarters of the slots, 0.9
    (12, 320, 250.0, 4.0, (64, 64, 29), (4.0, 4.0, 1.8181818), (0, 1, 1)),  # 2.1
    (9, 384, 250.0, 4.0, (128, 128, 12), (2.5, 2.5, 4.0), (1, 1, 1)),       # 0.63 of the slots, 0.1
    (9, 384, 250.0, 4.0, (64, 64, 15), (4.0, 4.0, 3.0), (0, 1, 1)),         # 0.7
    (7, 384, 250.0, 4.0, (64, 64, 13), (4.0, 4.0, 2.4), (0, 1, 0)),         # one warp per track, 1.0
    (64, 640, 410.0, 3.2, (320, 320, 144), (1.5, 1.5, 1.5), (1, 1, 1)),     # 2.3
    (64, 640, 410.0, 3.2, (320, 320, 128), (1.5, 1.5, 1.5), (0, 1, 0)),     # the same, 1 % clipped
])
def test_routes_by_fill_and_stops(rings, crystals, radius, pitch, size, voxel, routes):
    plan = capi.track_plan(ScannerSpec.ring(rings, crystals, radius, pitch),
                           ProjSpec(rings, crystals, 2 * rings - 1, crystals // 4 - 5), VolSpec.centred(size, voxel),
                           geometry=1)
    assert (plan.forward_on_tracks, plan.backward_on_tracks, plan.osem_on_tracks) == routes, (plan.stops, plan.general)

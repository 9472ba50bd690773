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
    assert plan.on_tracks and plan.ring_pairs == 85744 and plan.clipped > 0
    # a block's list of LORs for the general walk holds a place for each
    assert plan.block_tracks * plan.block_pairs * 4 <= plan.shared_bytes


def test_plan_rejects_what_the_projectors_reject():
    scanner, proj, vol = MANY_RINGS
    for bad in (dict(n_subsets=5), dict(n_subsets=2, subset=2), dict(block_size=48), dict(geometry=7)):
        with pytest.raises(capi.FirError):
            capi.track_plan(scanner, proj, vol, **bad)

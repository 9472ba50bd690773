"""Contexts of several host threads, whose volumes need different amounts of
shared memory above 48 KB, run their projections side by side."""
import os
import subprocess

import pytest

from fir_b200 import capi
from fir_b200.build import CXX, LIB_DIR, ROOT
from fir_b200.geometry import ProjSpec, ScannerSpec, VolSpec

PROGRAM = r"""
#include "fir_cuda.h"
#include <cuda_runtime.h>
#include <cstdio>
#include <string>
#include <thread>
#include <vector>

static int loop(int n, int calls, std::string* error)
{
  fir_scanner_desc sc{};
  sc.rsector_repeat = 128;
  sc.rsector_inner_radius = 400.0;
  sc.crystal_dims[2] = 4.0;
  sc.crystal_repeat[0] = 1;
  sc.crystal_repeat[1] = 8;
  sc.module_repeat[0] = sc.module_repeat[1] = 1;
  const fir_proj_desc pr{8, 128, 1, 15, 57};
  fir_vol_desc vol{n, n, 16, 2.0, 2.0, 2.0, -(n - 1.0), -(n - 1.0), 0.0, 1};
  fir_proj_info info;
  fir_proj_geometry(&pr, &info, nullptr);
  fir_ctx* c = nullptr;
  float *img = nullptr, *sino = nullptr;
  cudaStream_t st = nullptr;
  if (fir_ctx_create(&c, 0) != FIR_OK || fir_ctx_set_scanner(c, &sc) != FIR_OK ||
      cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&img, sizeof(float) * n * n * 16) != cudaSuccess ||
      cudaMalloc(&sino, sizeof(float) * info.n_bins) != cudaSuccess)
  {
    *error = "set-up failed";
    return 1;
  }
  cudaMemset(img, 0, sizeof(float) * n * n * 16);
  fir_ctx_set_stream(c, st);
  int failed = 0;
  for (int i = 0; i < calls; ++i)
  {
    if (fir_forward(c, &vol, img, &pr, sino) != FIR_OK)
    {
      ++failed;
      *error = fir_last_error();
    }
    if (i % 64 == 63)
    {
      cudaStreamSynchronize(st);
    }
  }
  if (fir_ctx_synchronize(c) != FIR_OK || fir_ctx_track_launch_count(c) < calls - failed)
  {
    ++failed;
    *error += " (end)";
  }
  fir_ctx_destroy(c);
  cudaFree(img);
  cudaFree(sino);
  return failed;
}

int main()
{
  const int sizes[4] = {320, 256, 320, 256};
  int failed[4];
  std::string error[4];
  std::vector<std::thread> ts;
  for (int k = 0; k < 4; ++k)
  {
    ts.emplace_back([&, k] { failed[k] = loop(sizes[k], 2000, &error[k]); });
  }
  for (auto& t : ts)
  {
    t.join();
  }
  int all = 0;
  for (int k = 0; k < 4; ++k)
  {
    std::printf("size %d: %d failed %s\n", sizes[k], failed[k], error[k].c_str());
    all += failed[k];
  }
  return all != 0;
}
"""


def sizes():
    scanner, proj = ScannerSpec.ring(8, 128, 400.0, 4.0), ProjSpec(8, 128, 15, 57)
    return [capi.track_plan(scanner, proj, VolSpec.centred((n, n, 16), (2.0, 2.0, 2.0))) for n in (320, 256)]


def test_plans_need_different_amounts():
    large, small = sizes()
    assert large.forward_on_tracks and small.forward_on_tracks
    assert 96 * 1024 >= large.shared_bytes > small.shared_bytes > 48 * 1024


@pytest.mark.gpu
def test_two_sizes_in_four_threads(tmp_path):
    src, exe = tmp_path / "loop.cc", str(tmp_path / "loop")
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run([CXX, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"), "-I", cuda + "/include", "-o", exe,
                    str(src), "-L", LIB_DIR, "-lfir_cuda", "-L", cuda + "/lib64", "-lcudart", "-lpthread",
                    "-Wl,-rpath," + LIB_DIR + ":" + cuda + "/lib64"], check=True)
    done = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr

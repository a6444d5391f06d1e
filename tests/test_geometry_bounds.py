"""Camera matrices on the host: translations of at most 2^30 voxels, so that the
kernels' integer positions cannot wrap; ordinary cameras keep theirs."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "niftyrec_gb300", "csrc")
PROGRAM = """
#include "et_geometry.h"
#include <cstdio>
#include <cmath>
using namespace nrgb;
template <class G> int bad(const std::vector<G>& all) {
  int n = 0;
  for (const G& g : all)
    for (int i = 0; i < 12; ++i) n += !(std::fabs(g.fwd[i]) <= 1073741824.0) + !(std::fabs(g.bwd[i]) <= 1073741824.0);
  return n;
}
int main() {
  Cameras c;
  c.n = 5;
  c.angles = {0, 0, 0.3f, 3.14159f, 0.1f, 3.14159f, 3.14159f, 1.f, 0, 0.2f, 0, 0, 0.2f, 0, 0};
  c.centers = {2e9f, -3e12f, 8e9f, 0, 9.5f, 0, 4e10f, -7e9f, 3e18f, 7.5f, 9.5f, -1e15f, 5e9f, -2e9f, 11.5f};
  const std::vector<CamGeom> g = camera_geometry(c);
  float m[16];
  rotation_matrix(m, 0.1f, 0.2f, 0, 9.5f, 7.5f, 11.5f, 0);
  int same = 1;
  for (int i = 0; i < 12; ++i) same &= m[i] == g[4].fwd[i];
  std::printf("%d %d %d\\n", bad(g), bad(camera_geometry64(c)), same);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_translations_are_bounded(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I" + CSRC, "-I" + os.path.join(cuda, "include"),
                    str(src), os.path.join(CSRC, "et_geometry.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["0", "0", "1"]

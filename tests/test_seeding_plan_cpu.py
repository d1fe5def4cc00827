"""The plan of the seeding search (cpm_internal.h voronoi_grid), compiled for
the host: where the rings are scanned in FP32 first, the slack of 3 ferr that
its bound carries lengthens a scan by at most one ring, whatever the sides.  On
long lattices it would have been hundreds, and the kernel would have run for
hours past the bound on a call's work."""
import os
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include "cpm_internal.h"
int main() {
  const int cases[][5] = {
      {2, 64, 64, 1, 40}, {2, 4096, 4096, 1, 167772}, {2, 1 << 20, 8, 1, 80000},
      {2, 600000, 3, 1, 900000}, {2, 3, 600000, 1, 900000}, {2, 1 << 24, 64, 1, 10000000},
      {2, 1 << 28, 4, 1, 10000000}, {2, 700000000, 3, 1, 1000}, {3, 256, 256, 256, 33554},
      {3, 3, 3, 1 << 27, 20000000}};
  for (auto& c : cases) {
    const int n[3] = {c[1], c[2], c[3]};
    const gpucpm::VoronoiGrid vg = gpucpm::voronoi_grid(c[0], n, c[4]);
    printf("%d %.6g %.6g\n", vg.single ? 1 : 0, (double)vg.ferr, vg.wmin);
  }
}
"""


def test_fp32_search_takes_one_ring_more_at_most(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'gpu-cpm_gb300' / 'csrc'}",
                    f"-I{cuda}/include", str(src), "-o", str(exe)], check=True)
    rows = [line.split() for line in
            subprocess.run([str(exe)], check=True, capture_output=True,
                           text=True).stdout.splitlines()]
    assert len(rows) == 10
    extra = [3 * float(ferr) / float(w) for _, ferr, w in rows]
    assert all(e <= 1.0 for (single, _, _), e in zip(rows, extra) if single == "1")
    assert max(extra) > 200  # 2^28 x 4
    # ordinary sides keep the FP32 search; in the others a bucket is as narrow
    # as the short side
    assert [single for single, _, _ in rows] == list("1110000010")

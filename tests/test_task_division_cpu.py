"""The sweep's division of a task's number by the tasks of a row
(cpm_internal.h), compiled for the host: exact over its range, and no division
by zero for a replica that has no columns of targets in a slot of its batch
(even nx, in the slots of the last column of odd ones)."""
import os
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include "cpm_internal.h"
using namespace gpucpm;
int main(int argc, char** argv) {
  volatile int none = 0;
  if (task_reciprocal(none) == 0) return 2;
  const uint32_t top = (1u << 31) - 1;
  for (uint32_t d : {1u, 2u, 3u, 5u, 31u, 32u, 33u, 64u, 127u, 1000u, 65535u, 65536u, 1u << 25,
                     (1u << 25) + 1, top})
    for (uint32_t base : {0u, d, 2 * d, top / 2, top / d * d, top})
      for (int o = -3; o <= 3; ++o) {
        const uint32_t n = base + (uint32_t)o;
        if (n > top) continue;
        uint32_t rem;
        const uint32_t q = task_quotient(n, d, task_reciprocal((int)d), rem);
        if (q != n / d || rem != n % d) {
          printf("%u / %u: %u, %u\n", n, d, q, rem);
          return 1;
        }
      }
  return 0;
}
"""


def test_task_division(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=integer-divide-by-zero",
                    "-fno-sanitize-recover=all", f"-I{ROOT / 'gpu-cpm_gb300' / 'csrc'}",
                    f"-I{cuda}/include", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

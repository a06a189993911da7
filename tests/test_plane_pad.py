"""The bank-conflict padding of the stash sweep's geometry arrays (fsg_internal.h choose_plane_pad), by a host
program compiled with nvcc from the library's own header: the same pad as a plain search over every probe
the stash kernel takes, in less than half its time (a call of fsg_simus sets it up twice)."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include "fsg_common.cuh"
#include "fsg_internal.h"
static int plain(int E, int U, int gn, int st) {
  const int pitch = st + 1;
  int best_pad = 0, best_cost = 1 << 30;
  for (int pad = 0; pad < 32; ++pad) {
    const int plane = E * pitch + pad;
    int cost = 0;
    for (int i = 0; i < fsg::kSrcPerThread; ++i) {
      int count[32] = {0}, worst = 0;
      for (int l = 0; l < 32; ++l) {
        const int g = l % gn, pt = l / gn, src = g + gn * i;
        if (src >= E * U) continue;
        const int word = (src % U) * plane + (src / U) * pitch + pt;
        const int c = ++count[word % 32];
        if (c > worst) worst = c;
      }
      cost += worst;
    }
    if (cost < best_cost) { best_cost = cost; best_pad = pad; }
  }
  return best_pad;
}
int main() {
  using clock = std::chrono::steady_clock;
  double t[2] = {0, 0};
  int n = 0;
  for (int U = 1; U <= 8; ++U)
    for (int E = 1; E <= (U > 4 ? 64 : 32); ++E)
      for (int gn = 4; gn <= 32; gn *= 2) {
        const int st = fsg::kThreads / gn;
        const auto a = clock::now();
        const int p = plain(E, U, gn, st);
        const auto b = clock::now();
        const int q = fsg::choose_plane_pad(E, U, gn, st);
        const auto c = clock::now();
        if (p != q) { printf("E %d U %d gn %d: %d, plain search %d\n", E, U, gn, q, p); return 1; }
        t[0] += std::chrono::duration<double>(b - a).count();
        t[1] += std::chrono::duration<double>(c - b).count();
        ++n;
      }
  printf("ok %d %g %g\n", n, 1e6 * t[0] / n, 1e6 * t[1] / n);
  return t[1] < 0.5 * t[0] ? 0 : 1;
}
"""


def test_plane_pad_equals_the_plain_search(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src = tmp_path / "pad.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "pad"
    csrc = ROOT / "fastsimus_gb300" / "csrc"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", f"-I{csrc}",
                        f"-I{ROOT / 'include'}", str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout

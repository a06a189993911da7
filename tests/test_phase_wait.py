"""The bounded waits' parity (fsg_tc.cuh phase_pass, used by tc_kernel): a host program compiled with nvcc
from the library's own header plays an mbarrier whose phases complete late.  After a wait that gave up, the
final wait before the tensor memory is released must stand on the phase that is still outstanding (the
opposite parity counts as complete and would return at once)."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdio>
#include "fsg_tc.cuh"
// An mbarrier: `done` phases have completed.  A test of parity p succeeds while the phase in
// progress (number `done`) has the other parity.
struct Barrier {
  int done = 0;
  bool test(uint32_t p) const { return (uint32_t)(done & 1) != p; }
};
int main() {
  for (int before = 0; before < 5; ++before) {   // phases that complete in time
    for (int polls = 0; polls < 4; ++polls) {    // polls until the late phase completes, in the final wait
      Barrier b;
      uint32_t parity = 0;
      for (int k = 0; k < before; ++k) {
        if (fsg::tc::phase_pass(parity, [&](uint32_t p) { return b.test(p); })) { printf("early\n"); return 1; }
        ++b.done;
        if (!fsg::tc::phase_pass(parity, [&](uint32_t p) { return b.test(p); })) { printf("missed\n"); return 1; }
      }
      // the phase in flight gives up, twice; then the final wait polls until it completes
      for (int k = 0; k < 2; ++k)
        if (fsg::tc::phase_pass(parity, [&](uint32_t p) { return b.test(p); })) { printf("gave up, yet passed\n"); return 1; }
      int n = 0;
      const bool ok = fsg::tc::phase_pass(parity, [&](uint32_t p) {
        for (; n < 10; ++n) {
          if (b.test(p)) return true;
          if (n == polls) ++b.done;
        }
        return false;
      });
      if (!ok || n != polls + 1) { printf("final wait: ok %d after %d polls, want %d\n", (int)ok, n, polls + 1); return 1; }
    }
  }
  printf("ok\n");
  return 0;
}
"""


def test_a_wait_that_gave_up_keeps_its_phase(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src = tmp_path / "phase.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "phase"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'fastsimus_gb300' / 'csrc'}", "-o", str(exe), str(src)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout

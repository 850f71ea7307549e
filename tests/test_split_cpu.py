"""Host-side parts of the digit GEMM (csrc/split_gemm.h), without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# One tile's MMA thread and one reading warp.  A barrier is the number of its
# completed phases; a wait for parity p passes when the phase in hand has the
# other parity.  `shared`: the lists use the same columns, so that the MMA thread
# waits for the reader between them.  Every order of commits and looks is walked:
# no wait may pass before its list is complete, and with both lists complete the
# reader has to come through.
WAITS = r"""
#include <cstdio>
#include "split_gemm.h"
using rbc::split_acc_wait;
static bool passes(int list, int done) {
  const auto w = split_acc_wait(list);
  int phases = 0;
  for (int l = 0; l < done; l++) phases += split_acc_wait(l).barrier == w.barrier;
  return (unsigned)(phases & 1) != w.parity;
}
static int walk(bool shared, int done, int reader) {
  int bad = 0;
  if (reader < 2) {
    if (passes(reader, done)) {
      if (done <= reader) bad += printf("shared %d: list %d read early\n", shared, reader);
      else bad += walk(shared, done, reader + 1);
    } else if (done == 2) {
      bad += printf("shared %d: list %d is never read\n", shared, reader);
    }
  }
  if (done < 2 && (done == 0 || !shared || reader >= 1)) bad += walk(shared, done + 1, reader);
  return bad;
}
int main() { return walk(true, 0, 0) + walk(false, 0, 0) != 0; }
"""

# A tile that gives up waits for the commits below before it frees its memory.
# Whatever chunk it gave up at, the last MMA issued has to be under one of them.
DRAIN = r"""
#include <algorithm>
#include <cstdio>
#include "split_gemm.h"
int main() {
  int bad = 0;
  for (int stages = 2; stages <= 3; stages++)
    for (int nc0 = 1; nc0 <= 20; nc0++)
      for (int nc1 = 0; nc1 <= nc0; nc1++)
        for (int issued = 1, total = nc0 + nc1; issued <= total; issued++) {
          int covered = 0;  // chunks whose MMAs a commit covers
          for (int c = 0; c < issued; c++)
            if (c + stages < total || c + 1 == nc0 || c + 1 == total) covered = c + 1;
          if (rbc::split_drain_commit(issued, total)) covered = issued;
          if (covered < issued)
            bad += printf("%d + %d chunks: gave up after %d, waits for %d\n", nc0, nc1, issued, covered);
        }
  return bad != 0;
}
"""


def _run(tmp_path, text):
    cxx = shutil.which("g++")
    inc = next((d for d in ("/usr/local/cuda/include", "/usr/local/cuda/targets/sbsa-linux/include")
                if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(text)
    subprocess.run([cxx, "-std=c++17", "-I", inc, "-I", os.path.join(ROOT, "rustpde_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_no_accumulator_wait_is_lost(tmp_path):
    _run(tmp_path, WAITS)


def test_a_tile_that_gives_up_waits_for_its_products(tmp_path):
    _run(tmp_path, DRAIN)

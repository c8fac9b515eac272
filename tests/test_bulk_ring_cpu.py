"""CPU test of the ring of bulk copies (bulk_ring.h) on a model of its barriers: after any number of issued copies,
waiting for the copies that it lists as open lasts until every one of them has landed, in whatever state the
barriers are, and does not wait for one that was never issued."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MODEL = r"""
#include <cstdio>
#include "bulk_ring.h"

template <int R>
int check() {
  using Ring = BulkRing<R>;
  for (int issued = 0; issued <= 6 * R + 1; ++issued) {
    // a stage is filled again only after its last copy landed: any subset of the last R may be in flight
    const int open = issued < R ? issued : R;
    for (unsigned flying = 0; flying < (1u << open); ++flying) {
      int phase[R] = {};  // completed phases of each stage's barrier
      for (int i = 0; i < issued; ++i) {
        const int back = issued - 1 - i;
        if (back >= R || !((flying >> back) & 1u)) ++phase[i % R];
      }
      // a wait for parity p returns once the phase of that parity has completed, i.e. is not the current one
      auto passes = [&](int i) { return (unsigned)(phase[Ring::stage(i)] & 1) != Ring::parity(i); };
      bool all = true;
      int waited = 0;
      for (int i = Ring::first_open(issued); i < issued; ++i, ++waited) all = all && passes(i);
      if (all != (flying == 0) || waited != open) {
        std::printf("R %d issued %d flying %x\n", R, issued, flying);
        return 1;
      }
    }
  }
  return 0;
}

int main() { return check<1>() | check<2>() | check<3>() | check<8>(); }
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_open_copies(tmp_path):
    src = tmp_path / "ring.cpp"
    src.write_text(MODEL)
    exe = str(tmp_path / "ring")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nomad_b200", "csrc", "cuda"), str(src), "-o", exe],
                   check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout

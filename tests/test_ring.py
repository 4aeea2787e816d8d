"""Which barrier phase the latest use of each stage of a ring completes (csrc/ring.h): what a
kernel that gives up waits for before it retires.  Compiled for the host and compared with
barriers whose phases are counted."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "chord_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "ring.h"

// Waiting on `parity` ends once a phase of that parity has completed and the next has not.
static bool passes(uint32_t completed, uint32_t parity) { return (completed & 1u) != parity; }

int main() {
  for (uint32_t stages = 1; stages <= 7; ++stages) {
    chord::StageCursor cur;
    std::vector<uint32_t> uses(stages, 0);
    for (int issued = 0; issued < 40; ++issued) {
      for (uint32_t i = 0; i < stages; ++i) {
        const uint32_t parity = cur.last_phase(i);
        if (!passes(uses[i], parity)) return std::printf("lands, yet waited for: %u %d %u\n", stages, issued, i), 1;
        if (uses[i] > 0 && passes(uses[i] - 1, parity)) return std::printf("in flight, yet not waited for: %u %d %u\n", stages, issued, i), 1;
      }
      ++uses[cur.s];
      cur.advance(stages);
    }
  }
  return 0;
}
"""


def test_last_phase_of_every_stage(tmp_path):
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "ring.cc").write_text(PROGRAM)
    binary = tmp_path / "ring"
    subprocess.run([compiler, "-std=c++17", f"-I{CSRC}", str(tmp_path / "ring.cc"), "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout

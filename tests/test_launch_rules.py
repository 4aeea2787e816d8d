"""The rules of launches in csrc/register_split.h and csrc/align_rules.h, compiled for the host."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "chord_b200" / "csrc"

REGISTERS = r"""
#include "register_split.h"
using chord::register_split_fits;

// Four warps go down to 56 registers, sixteen up to 104: 1888 of the 20 * 96 there are.
static_assert(register_split_fits(96, 4, 56, 16, 104), "");
static_assert(register_split_fits(95, 4, 56, 16, 104), "handed out in eights");
static_assert(!register_split_fits(88, 4, 56, 16, 104), "1888 of 1760");
static_assert(!register_split_fits(80, 4, 56, 16, 104), "");
static_assert(!register_split_fits(96, 4, 64, 16, 112), "2048 of 1920");
static_assert(!register_split_fits(48, 4, 56, 16, 40), "a share that goes the other way");
int main() { return 0; }
"""


def _run(tmp_path, source):
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "rules.cc").write_text(source)
    binary = tmp_path / "rules"
    built = subprocess.run([compiler, "-std=c++17", f"-I{CSRC}", str(tmp_path / "rules.cc"), "-o", str(binary)],
                           capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    return subprocess.run([str(binary)], capture_output=True, text=True)


def test_registers_of_the_decode_kernels_warps(tmp_path):
    assert _run(tmp_path, REGISTERS).returncode == 0


ALIGNMENT = r"""
#include <cstdio>
#include <initializer_list>
#include "align_rules.h"
using namespace chord;

int main() {
  for (int64_t experts = 1; experts <= 2048; ++experts) {
    for (int64_t numel : {0, 1, 512, 513, 1024, 1025, 2048, 2049, 4095, 4096, 32768, 1 << 30}) {
      const bool counters_fit = moe_align_smem_bytes(experts, kAlignWarps) <= kAlignMaxSmem;
      const AlignKernel with = align_kernel(numel, experts, true), without = align_kernel(numel, experts, false);
      const AlignKernel one_cta = numel <= 512 || numel <= experts ? AlignKernel::kShort : AlignKernel::kBatches;
      // no cluster where the device cannot place one, and then the same CTA as elsewhere
      if (without != one_cta) return std::printf("without a cluster: %lld ids, %lld experts\n", (long long)numel, (long long)experts), 1;
      if (with != (numel >= 4096 && counters_fit ? AlignKernel::kCluster : one_cta)) return std::printf("with: %lld ids, %lld experts\n", (long long)numel, (long long)experts), 1;
      if (moe_align_smem_bytes(experts, kAlignWarpsFew) > kAlignMaxSmem) return std::printf("%lld experts\n", (long long)experts), 1;
    }
  }
  return 0;
}
"""


def test_alignment_without_a_cluster(tmp_path):
    done = _run(tmp_path, ALIGNMENT)
    assert done.returncode == 0, done.stdout

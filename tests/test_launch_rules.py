"""The rules of launches in csrc/launch_rules.h, compiled for the host."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "chord_b200" / "csrc"

REGISTERS = r"""
#include "launch_rules.h"
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

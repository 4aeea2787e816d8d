"""The recorded DRAM traffic of the decode kernel counts only while every file that the kernel is
compiled from is the one it was captured on."""

import hashlib
import json
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "chord_b200" / "csrc"


def _sources(name, seen):
    """`name` and the files of the same folder that it includes, directly or not."""
    if name not in seen:
        seen.add(name)
        for included in re.findall(r'#include "([^"/]+)"', (CSRC / name).read_text()):
            _sources(included, seen)
    return seen


@pytest.mark.parametrize("changed", range(3))
def test_a_change_to_any_file_ends_the_record(tmp_path, monkeypatch, changed):
    import bench

    monkeypatch.setattr(bench, "ROOT", tmp_path)
    (tmp_path / "profiles").mkdir()
    names = ["a.cuh", "b.cuh", "c.h"]
    for name in names:
        (tmp_path / name).write_text(name)
    digest = hashlib.sha256(b"".join((tmp_path / name).read_bytes() for name in names)).hexdigest()
    record = {"source": names, "source_sha256": digest, "dram_bytes_per_step": 1}
    (tmp_path / "profiles" / "w4a16_decode_kernel_traffic.json").write_text(json.dumps(record))
    assert bench.recorded_traffic() == record
    (tmp_path / names[changed]).write_text("another")
    assert bench.recorded_traffic() is None
    (tmp_path / names[changed]).unlink()
    assert bench.recorded_traffic() is None


def test_the_committed_record_names_every_file_of_the_kernel():
    record = json.loads((ROOT / "profiles" / "w4a16_decode_kernel_traffic.json").read_text())
    named = {Path(name).name for name in record["source"]}
    assert named == _sources("w4a16_decode.cuh", set())
    assert all((ROOT / name).exists() for name in record["source"])

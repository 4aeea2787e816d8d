"""The integer-argument call module gives what ctypes gives, and refuses what it cannot pass."""

import pytest

from chord_b200 import _lib


def test_native_calls_agree_with_ctypes(native_lib):
    native = _lib.native()
    for routed in (0, 1, 300, 2000, 10000):
        assert native.chord_b200_indexed_block_m(4096, 7168, 48, routed) == \
            native_lib.chord_b200_indexed_block_m(4096, 7168, 48, routed)
    arguments = (1 << 40,) * 4 + (100, 1 << 40, 10, 1 << 40, 1 << 40, 1 << 40, 1024, 1 << 40, 100, 1 << 40,
                                  0, 4096, 7168, 48, 8, 16, 0)
    assert native.chord_b200_indexed(*arguments) == native_lib.chord_b200_indexed(*arguments) == 1
    with pytest.raises(ValueError, match="m=0"):
        _lib.check(native.chord_b200_indexed(*arguments))


needs_module = pytest.mark.skipif(_lib._call is None, reason="the call module was not built")


@needs_module
def test_arguments_that_are_no_integers(native_lib):
    with pytest.raises(TypeError):
        _lib.native().chord_b200_masked_tile_m("8")
    with pytest.raises(TypeError):
        _lib.native().chord_b200_masked_tile_m(None)
    with pytest.raises(TypeError):
        _lib.native().chord_b200_masked_tile_m(8.0)
    with pytest.raises(OverflowError):
        _lib.native().chord_b200_masked_tile_m(1 << 70)


@needs_module
@pytest.mark.parametrize("count", [0, 2, 3, 5, 25])
def test_wrong_numbers_of_arguments(native_lib, count):
    with pytest.raises(TypeError, match=f"takes 4 arguments.*got {count}"):
        _lib.native().chord_b200_indexed_block_m(*range(count))


def test_none_is_the_null_pointer(native_lib):
    for lib in (_lib.native(), native_lib):
        assert lib.chord_b200_silu_mul(None, 1 << 40, 4, 64, None) == 1
        assert "null tensor pointer" in _lib.last_error()


def test_module_counts_as_part_of_the_build(native_lib, monkeypatch, tmp_path):
    from chord_b200 import build

    assert build.is_fresh()
    monkeypatch.setattr(build, "_call_module_path", lambda: tmp_path / "_call.so")
    if build._call_compiler() is not None:
        assert not build.is_fresh()
    monkeypatch.setattr(build, "_call_compiler", lambda: None)
    assert build.is_fresh()


def test_failed_module_build_is_reported(native_lib, monkeypatch, tmp_path):
    from chord_b200 import build

    stale = tmp_path / "_call.so"
    stale.write_bytes(b"of an earlier version")
    monkeypatch.setattr(build, "_call_module_path", lambda: stale)
    monkeypatch.setattr(build, "_call_compiler", lambda: ["false"])
    with pytest.warns(UserWarning, match="ctypes"):
        build._build_call_module()
    assert not stale.exists()

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


def test_arguments_that_are_no_integers(native_lib):
    if _lib._call is None:
        pytest.skip("the call module was not built")
    with pytest.raises(TypeError):
        _lib.native().chord_b200_masked_tile_m("8")
    with pytest.raises(OverflowError):
        _lib.native().chord_b200_masked_tile_m(1 << 70)
    with pytest.raises(TypeError, match="at most 24"):
        _lib.native().chord_b200_masked_tile_m(*range(25))

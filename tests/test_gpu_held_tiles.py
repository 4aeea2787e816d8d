"""Tiles that are held in registers while they are stored (two weight blocks per tile, more than
64 tokens, or CTA pairs) and the block sizes next to them: more tiles than CTAs, so that whole
tiles and stream-K slices both occur, and row counts around the 16-token chunks of the epilogue."""

import pytest
import torch

from tests.cases import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_m,n,k", [(64, 5120, 192), (72, 5120, 64), (80, 5120, 192), (120, 5120, 320), (128, 5120, 128),
                                         (128, 5248, 192), (144, 2560, 2048), (208, 2560, 2112), (256, 2560, 2048)])
@pytest.mark.parametrize("groups", [2, 4])
def test_whole_tiles(device, block_m, n, k, groups):
    import chord_b200
    from chord_b200 import _lib

    counts = (1, 15, 16, 17, block_m - 1, block_m, block_m + 1, 2 * block_m)
    codes, scale = make_weights(len(counts), n, k, seed=block_m + k)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    total, ids, experts, row = sum(counts), [], [], 0
    for e, c in enumerate(counts):
        blocks = -(-c // block_m)
        ids += list(range(row, row + c)) + [total] * (blocks * block_m - c)
        experts += [e] * blocks
        row += c
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    x = torch.randn((total, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16).to(device)
    out = torch.full((total + 1, n), -7.0, dtype=torch.bfloat16, device=device)
    _lib.set_option("dequant_groups", groups)
    try:
        chord_b200.indexed(x, w, as_int(ids), as_int(experts), as_int([len(ids)]), 1, outputs=out[:total], block_m=block_m)
    finally:
        _lib.set_option("dequant_groups", 2)
    chord_b200.check_status(device)
    row = 0
    for e, c in enumerate(counts):
        wd = ((codes[e] - 8).to(torch.bfloat16) * scale[e].repeat_interleave(32, 1)).to(device).double()
        xe = x[row:row + c].double()
        ref = xe @ wd.T
        # per K16 step four units in the last place of the FP32 sum (2^-22 of the absolute
        # products), as much for stream-K partials, one BF16 rounding
        limit = 1.01 * (ref.abs() * 2.0 ** -8 + (k / 16 + 2) * 2.0 ** -22 * (xe.abs() @ wd.abs().T))
        assert bool(((out[row:row + c].double() - ref).abs() <= limit).all())
        row += c
    assert bool((out[total] == -7.0).all())

"""`contiguous` with more 128-row blocks than a warp merges at a time: runs of every length that
cross the 32-block boundaries, blocks of no expert between them, on 128-row tiles (short K) and on
the two launches of left-over blocks and pairs (K >= 2048)."""

import pytest
import torch

from tests.cases import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [128, 2048])
@pytest.mark.parametrize("tile", [0, 256])
@pytest.mark.parametrize("runs", [(1,) * 40, (30, 3, 1, 31, 2), (31, 2, 33), (32, 32, 1), (5, 0, 27, 0, 0, 4, 1, 6, 25)])
def test_runs_across_the_merge_width(device, runs, k, tile):
    import chord_b200
    from chord_b200 import _lib

    n, experts = 256, len(runs)
    g = torch.Generator().manual_seed(sum(runs) + k)
    codes, scale = make_weights(experts, n, k, seed=k)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    index = []
    for e, blocks in enumerate(runs):
        if blocks == 0:
            index += [-1] * 128  # a block of no expert
            continue
        short = int(torch.randint(0, 128, (1,), generator=g))
        index += [e] * (128 * blocks - short) + [-1] * short
    m_indices = torch.tensor(index, dtype=torch.int32)
    x = torch.randn((len(index), k), generator=g).to(torch.bfloat16)
    x[m_indices < 0] = 0
    out = torch.full((len(index), n), -7.0, dtype=torch.bfloat16, device=device)
    _lib.set_option("contiguous_tile", tile)
    try:
        chord_b200.contiguous(x.to(device), w, m_indices.to(device), outputs=out)
    finally:
        _lib.set_option("contiguous_tile", 0)
    chord_b200.check_status(device)
    block_expert = m_indices[::128]
    assert bool((out.view(-1, 128, n)[(block_expert < 0).to(device)] == -7.0).all())
    for e in range(experts):
        rows = (block_expert.repeat_interleave(128) == e).to(device)
        wd = ((codes[e] - 8).to(torch.bfloat16) * scale[e].repeat_interleave(32, 1)).to(device).double()
        xe = x.to(device)[rows].double()
        ref = xe @ wd.T
        # per K16 step four units in the last place of the FP32 sum (2^-22 of the absolute
        # products), as much for stream-K partials, one BF16 rounding
        limit = 1.01 * (ref.abs() * 2.0 ** -8 + (k / 16 + 2) * 2.0 ** -22 * (xe.abs() @ wd.abs().T))
        assert bool(((out[rows].double() - ref).abs() <= limit).all())

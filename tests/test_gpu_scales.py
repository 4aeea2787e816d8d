"""Scales on both sides of the two dequantisations (|scale| < 2 and any): small and large ones, of
either sign, zero, and single large ones among small ones, in every kernel that dequantises."""

import pytest
import torch

from tests.cases import make_weights
from tests.test_gpu_decode_tiles import _assert_close, _dequant, _routing, _sum_bound

pytestmark = pytest.mark.gpu


def _scales(kind, scale, g):
    sign = (torch.randint(0, 2, scale.shape, generator=g) * 2 - 1).to(torch.bfloat16)
    if kind == "signed":
        return scale * sign
    if kind == "edge":  # 2 - one unit in the last place, 2, and zeros
        pick = torch.randint(0, 3, scale.shape, generator=g)
        return torch.tensor([1.9921875, 2.0, 0.0], dtype=torch.bfloat16)[pick] * sign
    if kind == "large":
        return (torch.rand(scale.shape, generator=g) * 1e4 + 2).to(torch.bfloat16) * sign
    if kind == "tiny":
        return scale * 2.0 ** -100
    one_in = torch.rand(scale.shape, generator=g) < 1 / 64  # "few": some warps see one
    return torch.where(one_in, torch.tensor(96.0, dtype=torch.bfloat16), scale)


@pytest.mark.parametrize("kind", ["signed", "edge", "large", "tiny", "few"])
@pytest.mark.parametrize("block_m,n,k", [(16, 256, 320), (32, 256, 320), (64, 256, 320), (128, 256, 320),
                                         (256, 256, 320), (256, 256, 2048)])
def test_scales(device, kind, block_m, n, k):
    import chord_b200

    counts = (1, min(block_m, 9), block_m)
    g = torch.Generator().manual_seed(block_m + k)
    codes, scale = make_weights(len(counts), n, k, seed=k)
    scale = _scales(kind, scale, g)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    total = sum(counts)
    x = torch.randn((total, k), generator=g).to(torch.bfloat16)
    out = chord_b200.indexed(x.to(device), w, *_routing(counts, block_m, device), 1, block_m=block_m).cpu()
    wd, row = _dequant(codes, scale), 0
    for e, c in enumerate(counts):
        xe = x[row:row + c].double()
        _assert_close(out[row:row + c], xe @ wd[e].T, _sum_bound(xe, wd[e]))
        row += c


@pytest.mark.parametrize("kind", ["edge", "few"])
@pytest.mark.parametrize("block_m", [16, 128])
def test_scales_fused(device, kind, block_m):
    import chord_b200
    from chord_b200.indexed_gemm import indexed_gate_up_silu

    n, k, counts = 512, 256, (1, 9, block_m)
    g = torch.Generator().manual_seed(block_m)
    codes, scale = make_weights(len(counts), n, k, seed=k)
    scale = _scales(kind, scale, g)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    total = sum(counts)
    x = (torch.randn((total, k), generator=g) / 256).to(torch.bfloat16)
    out = indexed_gate_up_silu(x.to(device), w, *_routing(counts, block_m, device), 1, block_m=block_m).cpu()
    wd, row = _dequant(codes, scale), 0
    for e, c in enumerate(counts):
        both = x[row:row + c].double() @ wd[e].T
        gate, up = both[:, :n // 2], both[:, n // 2:]
        sums = _sum_bound(x[row:row + c].double(), wd[e])
        # d silu <= 1.1, |silu(g)| <= |g|; the exponential and the division are good to 2^-20
        bound = 1.1 * sums[:, :n // 2] * up.abs() + gate.abs() * sums[:, n // 2:] + (gate * up).abs() * 2.0 ** -20
        _assert_close(out[row:row + c], gate / (1 + torch.exp(-gate)) * up, bound)
        row += c

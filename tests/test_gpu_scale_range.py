"""Scales from the whole range of their type: down to BF16's subnormals, on both sides of 2^-5, where
the kernels change from one dequantisation to the other, infinite and NaN."""

import pytest
import torch

from tests.cases import make_weights
from tests.test_gpu_decode_tiles import _assert_close, _dequant, _routing, _sum_bound

pytestmark = pytest.mark.gpu

N, K = 256, 2112  # 2112: stream-K slices, and a half-filled last stage


def _scales(kind, scale, g):
    sign = (torch.randint(0, 2, scale.shape, generator=g) * 2 - 1).to(torch.float64)
    if kind == "edge":  # 2^-5 less one unit in the last place, 2^-5, and zeros
        pick = torch.randint(0, 3, scale.shape, generator=g)
        value = torch.tensor([0.0311279296875, 0.03125, 0.0], dtype=torch.float64)[pick]
    elif kind == "tiny":  # the type's smallest numbers: weights that are subnormal themselves
        value = 2.0 ** (torch.rand(scale.shape, generator=g, dtype=torch.float64) * 16 - 133)
    elif kind == "huge":  # up to the largest whose weights are finite
        value = 2.0 ** (torch.rand(scale.shape, generator=g, dtype=torch.float64) * 8 + 117)
        value = torch.where(value > 2.0 ** 122, 2.0 ** torch.randint(122, 125, scale.shape, generator=g).double(), value)
    else:  # "mixed": every stage has scales on both sides of 2^-5
        value = 2.0 ** (torch.rand(scale.shape, generator=g, dtype=torch.float64) * 16 - 12)
    return (value * sign).to(torch.bfloat16)


@pytest.mark.parametrize("mixed", [False, True])  # True: scales that share a stage differ by orders of magnitude
@pytest.mark.parametrize("block_m", [16, 32, 128, 256])
def test_every_scale_and_code(device, block_m, mixed):
    """Every scale whose weights are finite, with every code: a row of zeros and a one picks the weight
    RN_bf16((code - 8) * scale) out, to the bit."""
    import chord_b200

    experts, n, k = 4, 256, 2048
    patterns = torch.arange(experts * n * (k // 32), dtype=torch.int32)
    if mixed:
        patterns = patterns[torch.randperm(patterns.numel(), generator=torch.Generator().manual_seed(1))]
    scale = patterns.to(torch.int16).view(torch.bfloat16).view(experts, n, k // 32)
    scale = torch.where(scale.float().abs() < 2.0 ** 125, scale, torch.zeros_like(scale))
    codes = (torch.arange(k, dtype=torch.int32) % 16).expand(experts, n, k).contiguous()
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    picks = [32 * g + c for g in range(k // 32) for c in range(16)]
    rows = len(picks)  # for each expert, a multiple of every block_m
    x = torch.zeros((experts * rows, k), dtype=torch.bfloat16)
    x[torch.arange(experts * rows), torch.tensor(picks * experts)] = 1.0
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    routing = (as_int(list(range(experts * rows))),
               as_int([e for e in range(experts) for _ in range(rows // block_m)]), as_int([experts * rows]))
    out = chord_b200.indexed(x.to(device), w, *routing, 1, block_m=block_m).cpu().view(experts, rows, n)
    want = _dequant(codes, scale)[:, :, picks].transpose(1, 2)
    assert torch.equal(out.double(), want)


@pytest.mark.parametrize("kind", ["edge", "tiny", "mixed", "huge"])
@pytest.mark.parametrize("block_m", [8, 16, 32, 64, 128, 256])
def test_range(device, kind, block_m):
    import chord_b200

    counts = (1, min(block_m, 23), block_m)
    g = torch.Generator().manual_seed(block_m)
    codes, scale = make_weights(len(counts), N, K, seed=block_m)
    scale = _scales(kind, scale, g)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((sum(counts), K), generator=g).to(torch.bfloat16)
    x = x * {"tiny": 2.0 ** 100, "huge": 2.0 ** -110}.get(kind, 1.0)  # results in the middle of the range
    out = chord_b200.indexed(x.to(device), w, *_routing(counts, block_m, device), 1, block_m=block_m).cpu()
    wd, row = _dequant(codes, scale), 0
    for e, c in enumerate(counts):
        xe = x[row:row + c].double()
        _assert_close(out[row:row + c], xe @ wd[e].T, _sum_bound(xe, wd[e]))
        row += c


@pytest.mark.parametrize("kind", ["tiny", "mixed", "huge"])
@pytest.mark.parametrize("block_m", [16, 128])
def test_range_fused(device, kind, block_m):
    import chord_b200
    from chord_b200.indexed_gemm import indexed_gate_up_silu

    n, k, counts = 512, 256, (1, 9, block_m)
    g = torch.Generator().manual_seed(block_m)
    codes, scale = make_weights(len(counts), n, k, seed=k)
    scale = _scales(kind, scale, g)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((sum(counts), k), generator=g).to(torch.bfloat16) * {"tiny": 2.0 ** 100, "huge": 2.0 ** -122}.get(kind, 2.0 ** -8)
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


@pytest.mark.parametrize("block_m", [16, 32, 128, 256])
def test_infinite_and_nan(device, block_m):
    """A weight row with an infinite or a NaN scale gives what FP64 gives, and no other row does."""
    import chord_b200

    counts = (1, min(block_m, 23), block_m)
    g = torch.Generator().manual_seed(block_m + 1)
    codes, scale = make_weights(len(counts), N, K, seed=block_m + 1)
    scale[:, 3, 5], scale[:, 70, K // 32 - 1], scale[:, 200, 0] = float("inf"), float("-inf"), float("nan")
    codes[:, 3, 160:192] = 9  # inf * x of one column of a sign each: infinite or NaN, as the signs of x are
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((sum(counts), K), generator=g).to(torch.bfloat16)
    x[::2, 160:192] = x[::2, 160:192].abs() + 1
    out = chord_b200.indexed(x.to(device), w, *_routing(counts, block_m, device), 1, block_m=block_m).cpu()
    wd, row = _dequant(codes, scale), 0
    others = [r for r in range(N) if r not in (3, 70, 200)]
    for e, c in enumerate(counts):
        xe, got = x[row:row + c].double(), out[row:row + c].double()
        ref = xe @ wd[e].T
        assert torch.equal(torch.isnan(got), torch.isnan(ref))
        assert torch.equal(torch.isinf(got), torch.isinf(ref)) and bool((got[torch.isinf(got)] > 0).all())
        we = wd[e][others]
        _assert_close(out[row:row + c][:, others], ref[:, others], _sum_bound(xe, we))
        row += c

"""Edges of the decode kernel (token tiles of at most 32 rows): every count of rows around
its 8-, 16- and 32-column variants, K with and without a half stage at the end, a K short
enough for one stage and long enough for stream-K slices, `masked`, and the fused gate_up."""

import pytest
import torch

from tests.cases import make_weights

pytestmark = pytest.mark.gpu

COUNTS = {8: (1, 7, 8), 16: (1, 8, 9, 15, 16), 32: (1, 8, 9, 16, 17, 24, 31, 32)}


def _dequant(codes, scale):
    """The weights the kernels multiply with: RN_bf16((code - 8) * scale)."""
    return ((codes - 8).to(torch.bfloat16) * scale.repeat_interleave(32, 2)).double()


def _sum_bound(x, w):
    """What FP32 sums may be off by: per K16 step (one instruction adds sixteen products to a
    sum) 2^-22 of the sum of the absolute products, four units in the last place, and as much
    for the additions of stream-K partials (at most one per eight 128-wide stages)."""
    return (x.shape[-1] / 16 + 2) * 2.0 ** -22 * (x.abs() @ w.abs().transpose(-1, -2))


def _assert_close(got, ref, bound):
    """One BF16 rounding of the result (2^-8 of it at most) plus `bound`; the 1 % is for the
    products of the two."""
    limit = 1.01 * (ref.abs() * 2.0 ** -8 + bound)
    assert bool(((got.double() - ref).abs() <= limit).all())


def _routing(counts, block_m, device):
    """One block per entry of `counts`, block b of expert b, its rows at the front."""
    total = sum(counts)
    ids, row = [], 0
    for c in counts:
        ids += list(range(row, row + c)) + [total] * (block_m - c)
        row += c
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    return as_int(ids), as_int(list(range(len(counts)))), as_int([len(ids)])


@pytest.mark.parametrize("block_m", [8, 16, 32])
@pytest.mark.parametrize("n,k", [(128, 64), (256, 192), (128, 2048), (384, 1088)])
def test_every_row_count(device, block_m, n, k):
    import chord_b200

    counts = COUNTS[block_m]
    codes, scale = make_weights(len(counts), n, k, seed=block_m + k)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    total = sum(counts)
    x = torch.randn((total, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    out = torch.full((total, n), -7.0, dtype=torch.bfloat16, device=device)
    chord_b200.indexed(x.to(device), w, *_routing(counts, block_m, device), 1, outputs=out, block_m=block_m)
    wd, row = _dequant(codes, scale), 0
    for e, c in enumerate(counts):
        xe = x[row:row + c].double()
        _assert_close(out[row:row + c].cpu(), xe @ wd[e].T, _sum_bound(xe, wd[e]))
        row += c


@pytest.mark.parametrize("expected_m", [8, 20])
@pytest.mark.parametrize("k", [64, 320, 1024])
def test_masked_row_counts(device, expected_m, k):
    import chord_b200

    counts = (0, 1, 8, 9, 16, 17, 32, 33, 48)
    n, max_m = 256, 48
    codes, scale = make_weights(len(counts), n, k, seed=k)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((len(counts), max_m, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    out = torch.full((len(counts) * max_m, n), -7.0, dtype=torch.bfloat16, device=device)
    chord_b200.masked(x.to(device), w, torch.tensor(counts, dtype=torch.int32, device=device), expected_m,
                      outputs=out)
    out, wd = out.cpu().view(len(counts), max_m, n), _dequant(codes, scale)
    for g, c in enumerate(counts):
        xe = x[g, :c].double()
        _assert_close(out[g, :c], xe @ wd[g].T, _sum_bound(xe, wd[g]))
        assert bool((out[g, c:] == -7.0).all())


@pytest.mark.parametrize("n,k", [(256, 128), (512, 2048)])
def test_fused_row_counts(device, n, k):
    import chord_b200
    from chord_b200.indexed_gemm import indexed_gate_up_silu

    counts = COUNTS[16]
    codes, scale = make_weights(len(counts), n, k, seed=k)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    total = sum(counts)
    x = torch.randn((total, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    out = indexed_gate_up_silu(x.to(device), w, *_routing(counts, 16, device), 1, block_m=16).cpu()
    wd, row = _dequant(codes, scale), 0
    for e, c in enumerate(counts):
        both = x[row:row + c].double() @ wd[e].T
        gate, up = both[:, :n // 2], both[:, n // 2:]
        sums = _sum_bound(x[row:row + c].double(), wd[e])
        # d silu <= 1.1, |silu(g)| <= |g|; the exponential and the division are good to 2^-20
        bound = 1.1 * sums[:, :n // 2] * up.abs() + gate.abs() * sums[:, n // 2:] + (gate * up).abs() * 2.0 ** -20
        _assert_close(out[row:row + c], gate / (1 + torch.exp(-gate)) * up, bound)
        row += c


def test_values_out_of_range_stay_in_their_row(device):
    """Infinite and NaN activations give what the general kernel gives, and nothing of them
    reaches other rows of the tile."""
    import chord_b200
    from chord_b200 import _lib

    n, k, counts = 128, 256, (6, 13)
    codes, scale = make_weights(len(counts), n, k, seed=5)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((sum(counts), k), generator=torch.Generator().manual_seed(6)).to(torch.bfloat16)
    clean = x.clone()
    x[2, 17], x[9, 100], x[11, 3] = float("inf"), float("-inf"), float("nan")
    routing = _routing(counts, 16, device)
    run = lambda v: chord_b200.indexed(v.to(device), w, *routing, 1, block_m=16).cpu()
    got, unspoiled = run(x), run(clean)
    _lib.set_option("decode_kernel", 0)
    try:
        general = run(x)
    finally:
        _lib.set_option("decode_kernel", 1)
    assert bool((torch.isnan(got) == torch.isnan(general)).all())
    assert bool((torch.isinf(got) == torch.isinf(general)).all())
    others = [r for r in range(sum(counts)) if r not in (2, 9, 11)]
    assert torch.equal(got[others], unspoiled[others])


def test_largest_activations(device):
    """Activations near the end of the type's range; the weights are small, so the sums are not."""
    import chord_b200

    n, k = 128, 256
    codes, scale = make_weights(1, n, k, seed=7)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.zeros((3, k), dtype=torch.bfloat16)
    x[0, 5], x[1, 40], x[2] = 3e38, -2e37, 1.0
    out = chord_b200.indexed(x.to(device), w, *_routing((3,), 16, device), 1, block_m=16).cpu()
    wd = _dequant(codes, scale)[0]
    assert bool(torch.isfinite(out).all())
    _assert_close(out, x.double() @ wd.T, _sum_bound(x.double(), wd))

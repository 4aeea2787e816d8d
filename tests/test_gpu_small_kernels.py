"""Edges of the kernels either side of the GEMMs: where the alignment kernel changes its shape
(4096 ids, counters beyond 160 KB, more than one batch of loads), remainders and alignment of
the packer, row lengths of SiLU*mul."""

import pytest
import torch

from oracle import w4a16_oracle as O
from tests.cases import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel", [1, 511, 4095, 4096, 4097, 16385, 40001])
@pytest.mark.parametrize("experts,total,base", [(48, 384, 96), (1, 2, 1), (1241, 1241, 0), (1242, 1300, 7), (2048, 2048, 0)])
def test_alignment_shapes(device, numel, experts, total, base):
    import chord_b200

    g = torch.Generator().manual_seed(numel + experts)
    topk = torch.randint(0, total, (numel, 1), generator=g, dtype=torch.int32)
    s, e, p = chord_b200.moe_align_block_size(topk.to(device), 16, experts, expert_base=base)
    rs, re, rp = O.align_routing_blocks(topk, 16, experts, base)
    count = int(p.item())
    assert count == int(rp)
    assert torch.equal(s.cpu()[:count], rs)
    assert torch.equal(e.cpu()[: count // 16], re)


@pytest.mark.parametrize("numel", [512, 513, 2048, 2049, 32767, 32768, 32769, 100000])
@pytest.mark.parametrize("experts,total,base,block_m", [(48, 384, 144, 128), (3, 3, 0, 8), (1, 400, 7, 16), (1279, 1280, 1, 8),
                                                        (1280, 1280, 0, 8)])
def test_alignment_batches_and_clusters(device, numel, experts, total, base, block_m):
    """One round and one batch of ids per warp and one more; the last number of experts whose
    counters let a cluster of CTAs align, and the next; experts of very uneven popularity."""
    import chord_b200

    g = torch.Generator().manual_seed(numel + experts)
    topk = (torch.rand((numel, 1), generator=g) ** 3 * total).to(torch.int32)
    s, e, p = chord_b200.moe_align_block_size(topk.to(device), block_m, experts, expert_base=base)
    rs, re, rp = O.align_routing_blocks(topk, block_m, experts, base)
    count = int(p.item())
    assert count == int(rp)
    assert torch.equal(s.cpu()[:count], rs)
    assert torch.equal(e.cpu()[: count // block_m], re)


def test_alignment_ids_outside_every_range(device):
    import chord_b200

    ids = torch.tensor([[-2**31, 2**31 - 1, -1, 5, 7, 8, 4]], dtype=torch.int32)
    s, e, p = chord_b200.moe_align_block_size(ids.to(device), 8, 3, expert_base=5)  # experts 5, 6, 7
    assert int(p.item()) == 16
    assert s.cpu()[:16].tolist() == [3] + [7] * 7 + [4] + [7] * 7
    assert e.cpu()[:2].tolist() == [0, 2]


@pytest.mark.parametrize("k", [64, 448, 512, 576, 1088])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_packer_remainders_and_scale_alignment(device, k, offset):
    import chord_b200

    codes, scale = make_weights(2, 256, k, seed=k + offset)
    buffer = torch.zeros(scale.numel() + offset, dtype=torch.bfloat16, device=device)
    view = buffer[offset:].view(scale.shape)  # 2-, 4- or 16-byte aligned
    view.copy_(scale)
    words = torch.from_numpy(O.pack_checkpoint_uint4(codes.numpy())).to(device)
    want = torch.from_numpy(O.repack_closed_form(codes.numpy()))
    for w in (chord_b200.pack_w4a16(words, view, packed=True), chord_b200.pack_w4a16(codes.to(device), view)):
        assert torch.equal(w.packed.cpu(), want)
        assert torch.equal(w.scale.cpu().view(torch.int16), O.permute_scale(scale).view(torch.int16))


@pytest.mark.parametrize("rows,inter", [(1, 8), (300, 8), (7, 24), (33, 264), (5, 2048), (3, 2056),
                                        (2, 32776)])
def test_silu_mul_row_lengths(device, rows, inter):
    """FP32 arithmetic within a few units of 2^-21, then one rounding to BF16 (2^-8 at most)."""
    import chord_b200

    x = torch.randn((rows, 2 * inter), generator=torch.Generator().manual_seed(inter)).to(torch.bfloat16)
    got = chord_b200.silu_mul(x.to(device)).cpu().double()
    gate, up = x[:, :inter].double(), x[:, inter:].double()
    want = gate / (1 + torch.exp(-gate)) * up
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -18)).all())


@pytest.mark.parametrize("block_m", [16, 64])
def test_silu_mul_is_the_fused_epilogue(device, block_m):
    """One function, wherever it is computed: with weights that pick single activations the FP32
    accumulators of gate_up hold BF16 values exactly, and the fused epilogue (an IEEE quotient in
    FP32, one rounding) and the separate kernel give the same bits.  Half of the gates are the two
    BF16 values whose quotient lies so close to a rounding boundary of some products that
    v * reciprocal(1 + e^-v) lands on the other side."""
    import chord_b200
    from chord_b200.indexed_gemm import indexed_gate_up_silu

    n, tokens = 256, 8192
    codes = torch.full((1, n, n), 8, dtype=torch.int32)
    codes[0].fill_diagonal_(9)
    w = chord_b200.pack_w4a16(codes.to(device), torch.ones((1, n, n // 32), dtype=torch.bfloat16, device=device))
    g = torch.Generator().manual_seed(3)
    x = torch.randn((tokens, n), generator=g).sign_() * torch.exp(torch.rand((tokens, n), generator=g) * 12 - 8)
    x[::4, :n // 2], x[1::4, :n // 2] = -15.0, 0.0004444122314453125
    x = x.to(torch.bfloat16).to(device)
    routing = (torch.arange(tokens, dtype=torch.int32, device=device),
               torch.zeros(tokens // block_m, dtype=torch.int32, device=device),
               torch.tensor([tokens], dtype=torch.int32, device=device))
    gate_up = chord_b200.indexed(x, w, *routing, 1, block_m=block_m)
    assert torch.equal(gate_up, x)
    fused = indexed_gate_up_silu(x, w, *routing, 1, block_m=block_m)
    assert torch.equal(chord_b200.silu_mul(gate_up), fused)


def test_silu_mul_of_zero_gates(device):
    """Vectors of zero gates keep the sign of the product and what 0 * inf and 0 * nan give."""
    import chord_b200

    up = torch.tensor([1.0, -1.0, 0.0, -0.0, float("inf"), float("nan"), 1e-40, -3e38], dtype=torch.bfloat16)
    for gates in ([0.0] * 8, [-0.0] * 8, [0.0, -0.0] * 4, [0.0] * 7 + [2.0]):
        gate = torch.tensor(gates, dtype=torch.bfloat16)
        got = chord_b200.silu_mul(torch.cat([gate, up]).view(1, 16).to(device)).cpu()[0].float()
        want = torch.nn.functional.silu(gate.float()) * up.float()
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        keep = ~torch.isnan(want)
        assert torch.equal(torch.signbit(got[keep]), torch.signbit(want[keep]))
        assert torch.allclose(got[keep], want[keep], rtol=2.0 ** -8, atol=0)


def test_silu_mul_extreme_gates(device):
    import chord_b200

    gate = torch.tensor([float("inf"), float("-inf"), float("nan"), 3e38, -3e38, -88.5, -87.0, 0.0], dtype=torch.bfloat16)
    x = torch.cat([gate, torch.ones_like(gate)]).view(1, 16)
    got = chord_b200.silu_mul(x.to(device)).cpu().float()[0]
    assert got[0] == float("inf") and torch.isnan(got[1]) and torch.isnan(got[2])
    assert got[3] > 2.9e38 and got[4] == 0 and -1e-35 < got[5] <= 0 and -2e-35 < got[6] < 0 and got[7] == 0


@pytest.mark.parametrize("expected_m,n,k", [(120, 256, 2048), (121, 256, 2048), (144, 512, 2112), (130, 384, 2048),
                                            (130, 256, 1984)])
def test_masked_tile_choice(device, expected_m, n, k):
    """Both sides of the line between 128- and 256-row tiles; counts below, at and above both."""
    import chord_b200

    counts, max_m = (0, 1, 127, 128, 129, 200, 256, 300), 300
    codes, scale = make_weights(len(counts), n, k, seed=k + expected_m)
    w = chord_b200.pack_w4a16(codes.to(device), scale.to(device))
    x = torch.randn((len(counts), max_m, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    out = torch.full((len(counts) * max_m, n), -7.0, dtype=torch.bfloat16, device=device)
    chord_b200.masked(x.to(device), w, torch.tensor(counts, dtype=torch.int32, device=device), expected_m, outputs=out)
    out = out.cpu().view(len(counts), max_m, n)
    wd = ((codes - 8).to(torch.bfloat16) * scale.repeat_interleave(32, 2)).float()
    for g, c in enumerate(counts):
        ref = x[g, :c].float() @ wd[g].T
        # FP32 sums in two orders (2^-22 of the absolute products per term's depth), one BF16 rounding
        bound = 2.0 ** -17 * (x[g, :c].float().abs() @ wd[g].abs().T)
        assert bool(((out[g, :c].float() - ref).abs() <= 1.01 * (ref.abs() * 2.0 ** -8 + bound)).all())
        assert bool((out[g, c:] == -7.0).all())

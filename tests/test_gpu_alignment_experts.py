"""The alignment with as many ids as experts and one more, where it changes from one round of loads
ahead to four, on one CTA of several rounds per warp."""

import pytest
import torch

from oracle import w4a16_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts", [513, 1024, 2048])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("block_m", [8, 64])
def test_as_many_ids_as_experts(device, experts, more, block_m):
    import chord_b200

    topk = torch.randint(0, experts, (experts + more, 1), generator=torch.Generator().manual_seed(experts), dtype=torch.int32)
    s, e, p = chord_b200.moe_align_block_size(topk.to(device), block_m, experts)
    rs, re, rp = O.align_routing_blocks(topk, block_m, experts, 0)
    count = int(p.item())
    assert count == int(rp)
    assert torch.equal(s.cpu()[:count], rs)
    assert torch.equal(e.cpu()[: count // block_m], re)

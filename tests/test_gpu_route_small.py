"""Routing of at most 1024 slots in one block (`route_small_kernel`): the layout rules, checked against a count on the host."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one slot; fewer than a warp; every lane and expert in use; an expert with more than a padded segment; many experts, most of them empty; one more
# slot than the block takes (three launches)
@pytest.mark.parametrize("slots,experts", [(1, 8), (31, 8), (1024, 128), (1000, 2), (37, 100), (1025, 32)])
def test_routing_layout(slots, experts):
    from gpt_moe_b200.ops import cuda_ops
    gen = torch.Generator().manual_seed(slots + experts)
    idx = (torch.rand(slots, 1, generator=gen) ** 2 * experts).long().clamp_(max=experts - 1)
    dest, src, seg, counts, tiles, meta = (t.cpu() for t in cuda_ops.ext().route(idx.cuda(), experts))
    want = torch.bincount(idx.view(-1), minlength=experts)
    assert torch.equal(counts.long(), want)
    padded = (want + 255) // 256 * 256
    ends = padded.cumsum(0)
    assert torch.equal(seg.long(), ends) and meta.tolist() == [int(ends[-1]) // 128, int(ends[-1])]
    rows = torch.full((int(ends[-1]),), -1)
    for e in range(experts):                       # slots of an expert in their order, then pad rows
        mine = (idx.view(-1) == e).nonzero().view(-1)
        first = int(ends[e] - padded[e])
        rows[first: first + len(mine)] = mine
        assert (tiles[first // 128: int(ends[e]) // 128] == e).all()
    assert torch.equal(src[: len(rows)].long(), rows)
    assert torch.equal(rows[dest.long()], torch.arange(slots))

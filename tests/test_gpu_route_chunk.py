"""The one-CTA route inversion at the edges of its range."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("Qb,Kb,tk", [(1, 1, 1), (1, 600, 1), (3, 513, 512), (1023, 16, 16), (1024, 16, 16), (8, 6144, 2047)])
def test_route_inversion_of_a_slice_in_one_chunk(Qb, Kb, tk):
    from simple_vsa_b200 import ops
    g = torch.Generator().manual_seed(Qb)
    H = 2
    selected = torch.rand(1, H, Qb, Kb, generator=g).topk(tk, dim=-1).indices.to(torch.int32)
    selected[0, 0, 0, 0] = Kb + 5                   # ids outside the table are dropped
    inverse, offsets, counts = (x.cpu() for x in ops.invert_routes(selected.to(DEV), Kb))
    for h in range(H):
        ids = selected[0, h].reshape(-1).long()
        query = torch.arange(Qb).repeat_interleave(tk)[ids < Kb]
        ids = ids[ids < Kb]
        want = torch.bincount(ids, minlength=Kb)
        assert torch.equal(counts[0, h].long(), want)
        assert torch.equal(offsets[0, h].long(), want.cumsum(0) - want)
        got = inverse[0, h][:ids.numel()].long()
        owner = torch.arange(Kb).repeat_interleave(want)
        assert torch.equal((owner * Qb + got).sort().values, (ids * Qb + query).sort().values)

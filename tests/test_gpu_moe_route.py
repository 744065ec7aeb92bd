"""Counting, planning and dispatch of the MoE layer at the edges of its work split."""

import pytest
import torch

from lplb_b200 import Planner, cube
from lplb_b200.models.moe import MoELayer

pytestmark = pytest.mark.gpu


# pairs: none, one, around one CTA's 256, one per thread on every SM, beyond the four that a thread
# keeps in registers; hidden: one partial 2 KB piece of a row, exactly one, several and a remainder
@pytest.mark.parametrize(
    "tokens,topk,hidden", [(0, 2, 256), (1, 1, 256), (255, 1, 1024), (257, 1, 1280), (4737, 8, 512), (20000, 8, 256)]
)
@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_every_pair_lands_in_its_experts_rows(tokens, topk, hidden, dtype):
    planner = Planner(cube(), 32 + 16, 32, 8, device="cuda")
    layer = MoELayer(planner, hidden, 128, topk, max_tokens=max(1, tokens))
    g = torch.Generator("cuda").manual_seed(tokens)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()
    w = torch.rand(tokens, topk, device="cuda", generator=g)
    for _ in range(2):  # the counters are left at zero
        phys = torch.randint(-1, 48, (tokens, topk), device="cuda", generator=g).to(dtype)
        layer.forward_physical(x, phys, w, upto=2)
        torch.cuda.synchronize()
        assert layer.check() == 0
        plan = layer.engine.plan().cpu().long()
        flat = phys.reshape(-1).long()
        rows = torch.bincount(flat[flat >= 0], minlength=48).cpu()
        assert torch.equal(plan[:48], rows) and torch.equal(plan[48:96], rows.cumsum(0) - rows)
        slot = layer.engine.pair_slot()[: flat.numel()].long()
        assert torch.equal(slot >= 0, flat >= 0)
        total = int(rows.sum())
        assert torch.equal(slot[slot >= 0].sort().values.cpu(), torch.arange(total))
        # on one rank return slots and receive rows are numbered alike
        assert torch.equal(layer.engine.recv_meta()[:total].cpu().long(), torch.arange(total))
        owner = torch.repeat_interleave(torch.arange(48), rows).cuda()
        pair = (slot >= 0).nonzero().reshape(-1)
        assert torch.equal(owner[slot[pair]], flat[pair])
        assert torch.equal(layer.engine.recv_x()[slot[pair]], x[pair // topk])


def test_out_of_range_physical_ids_are_counted_and_dropped():
    planner = Planner(cube(), 32 + 16, 32, 8, device="cuda")
    layer = MoELayer(planner, 256, 128, 2, max_tokens=8)
    phys = torch.tensor([[0, 48], [-1, -5], [47, 1]], device="cuda")
    layer.forward_physical(torch.ones(3, 256, device="cuda").bfloat16(), phys, torch.ones(3, 2, device="cuda"), upto=2)
    torch.cuda.synchronize()
    assert layer.engine.pair_slot()[:6].tolist() == [0, -1, -1, -1, 2, 1]
    assert int(layer.engine.status()[8 + 7]) == 2

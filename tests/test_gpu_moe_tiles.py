"""The grouped GEMMs at the edges of their tiles: received rows per expert, and barriers that come round."""

import pytest
import torch

from lplb_b200 import Planner, ring
from lplb_b200.models.moe import MoELayer

pytestmark = pytest.mark.gpu

# none; one; around a step of 32, a half of 128 rows and a tile of 256; two and three tiles with
# even and uneven shares; nine tiles
ROWS = [0, 1, 31, 32, 33, 127, 128, 129, 224, 225, 255, 256, 257, 288, 511, 513, 0, 769, 2049, 16]


# inter 128: two K blocks in the second GEMM, the fewest there are
@pytest.mark.parametrize("hidden,inter", [(256, 128), (768, 384)])
@pytest.mark.parametrize("send_ctas", [None, 0, 1, 15])  # None: stand-alone dispatch; odd counts become whole pairs
def test_every_row_count_of_an_expert(hidden, inter, send_ctas):
    planner = Planner(ring(2), 16 + 4, 16, 2, device="cuda", n_nodes=1)
    assert planner.n_routed_experts == len(ROWS)
    tokens = sum(ROWS)
    layer = MoELayer(planner, hidden, inter, 1, max_tokens=tokens)
    layer.engine.set_timeout_us(2e5)
    layer.fuse_dispatch, layer.send_ctas = send_ctas is not None, send_ctas or 0
    g = torch.Generator("cuda").manual_seed(hidden)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()
    for counts in (ROWS, ROWS[::-1]):
        owner = torch.repeat_interleave(torch.arange(len(ROWS)), torch.tensor(counts)).cuda()
        phys = owner[torch.randperm(tokens, device="cuda", generator=g)].unsqueeze(1)
        out = layer.forward_physical(x, phys, torch.ones(tokens, 1, device="cuda"))
        torch.cuda.synchronize()
        assert layer.check() == 0
        for slot in range(len(ROWS)):
            mine = phys[:, 0] == slot
            if not bool(mine.any()):
                continue
            gate, up, down = (w.float() for w in layer.logical_weights(int(planner.phy2log[slot])))
            xin = x[mine].float()
            act = torch.nn.functional.silu(xin @ gate.T) * (xin @ up.T)
            ref = act.bfloat16().float() @ down.T
            # two bf16 roundings (2^-9 each) of independent elements, plus activations that round
            # the other way in fp32 sums of another order: per row below 2^-7
            err = (out[mine].float() - ref).norm(dim=1) / ref.norm(dim=1)
            assert float(err.max()) < 2**-7, slot


# (experts, logical experts, rows per expert, hidden, inter, sender CTAs); every barrier and slot of the
# tile hand-out (16 slots), the ring (6 to 11 stages) and the accumulators comes round several times:
# 102 tiles of the first GEMM on one pair, of all sizes and of at most 32 rows; the second GEMM with its
# fewest K blocks on every pair, 28 x 124 tiles of at most 32 rows, 48 a pair
LONG = [
    (20, 16, ROWS, 256, 384, -2),
    (20, 16, [(7 * i) % 32 + 1 for i in range(20)], 256, 1280, -2),
    (128, 120, [i % 33 for i in range(128)], 7168, 128, None),
]


@pytest.mark.parametrize("case", range(len(LONG)))
def test_many_tiles_on_one_pair(case):
    experts, logical, rows, hidden, inter, senders = LONG[case]
    planner = Planner(ring(2), experts, logical, 2, device="cuda", n_nodes=1)
    assert planner.n_routed_experts == experts
    tokens = sum(rows)
    layer = MoELayer(planner, hidden, inter, 1, max_tokens=tokens)
    layer.engine.set_timeout_us(2e5)
    if senders is not None:  # all SMs but one pair only send
        layer.fuse_dispatch = True
        layer.send_ctas = torch.cuda.get_device_properties(0).multi_processor_count + senders
    g = torch.Generator("cuda").manual_seed(case)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()
    owner = torch.repeat_interleave(torch.arange(experts), torch.tensor(rows)).cuda()
    for _ in range(2):
        phys = owner[torch.randperm(tokens, device="cuda", generator=g)].unsqueeze(1)
        out = layer.forward_physical(x, phys, torch.ones(tokens, 1, device="cuda"))
        torch.cuda.synchronize()
        assert layer.check() == 0
        for slot in range(experts):
            mine = phys[:, 0] == slot
            if not bool(mine.any()):
                continue
            gate, up, down = (w.float() for w in layer.logical_weights(int(planner.phy2log[slot])))
            xin = x[mine].float()
            act = torch.nn.functional.silu(xin @ gate.T) * (xin @ up.T)
            ref = act.bfloat16().float() @ down.T
            err = (out[mine].float() - ref).norm(dim=1) / ref.norm(dim=1)
            assert float(err.max()) < 2**-7, slot  # the bound of the test above

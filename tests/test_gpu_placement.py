"""The placement kernel against the host balancer: the same tables, whatever the shape and the history."""

import pytest
import torch

from lplb_b200 import Planner, cube, ring, topology
from lplb_b200.mapping import build_mapping

pytestmark = pytest.mark.gpu

# (topology, LP groups, experts per rank, combined, nodes): one group, groups on one node, on fewer
# nodes, one per node, nodes that the groups do not divide over; one expert per rank; packs below
# and above a warp's 32 lanes; the largest number of experts
SHAPES = [
    (cube(), 1, 32, 1, 1), (cube(), 4, 8, 2, 1), (cube(), 4, 8, 1, 2), (cube(), 4, 9, 1, 4), (cube(), 2, 16, 1, 3),
    (ring(8), 2, 1, 1, 1), (ring(3), 5, 7, 2, 1), (topology.torus(8, 4), 1, 16, 1, 1), (topology.torus(8, 8), 1, 8, 1, 1),
    (ring(40), 4, 3, 1, 2), (ring(128), 1, 1, 1, 1), (cube(), 16, 64, 1, 4),
]


def _histories(n, seed):
    g = torch.Generator().manual_seed(seed)
    yield (torch.rand(n, generator=g) * 1e7).long()
    yield torch.randint(0, 3, (n,), generator=g)  # ties everywhere
    yield torch.zeros(n, dtype=torch.int32)
    yield torch.randint(-1000, 1000, (n,), generator=g, dtype=torch.int32)
    yield torch.randint(0, 2**40, (n,), generator=g)
    yield torch.randint(-100, 100, (n,), generator=g, dtype=torch.int8)
    yield torch.randint(0, 9, (2 * n,), generator=g)[::2]
    yield torch.rand(n, generator=g)  # not whole numbers: placed on the host


@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_same_tables_as_the_host(shape):
    r2o, n_group, ll, c, nodes = SHAPES[shape]
    ep = n_group * r2o.shape[0]
    n = ep * ll
    planner = Planner(r2o, n + ep * r2o.shape[1] * c, n, ep, device="cuda", n_nodes=nodes)
    twin = Planner(r2o, n + ep * r2o.shape[1] * c, n, ep, device="cuda", n_nodes=nodes)
    idx = torch.randint(-1, n, (777, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(shape))
    for i, hist in enumerate([None, *_histories(n, shape)]):
        if n > 1024 and i not in (1, 2, 4):  # the host takes a second or so for these
            continue
        want = build_mapping(r2o, n_group, ll, c, hist, n_nodes=nodes)
        on_gpu = hist is not None and i % 2 == 0
        got = planner.update_redundancy_mapping(hist.cuda() if on_gpu else hist)
        for a, b in zip(got, (want.phy2log, want.log2phy, want.logcnt)):
            assert a.dtype == torch.int32 and torch.equal(a.cpu(), b), i
        assert torch.equal(planner.mapping.log2edge.cpu(), want.log2edge), i
        # the engine's own tables: the same routing as a planner that was handed the host's tables
        twin.load_state_dict(planner.state_dict())
        a, b = (p.run(idx, torch.zeros(1, dtype=torch.int32, device="cuda")) for p in (planner, twin))
        assert torch.equal(planner.last_probs, twin.last_probs)
        assert torch.equal(planner.count_workload(idx, 4)[0], twin.count_workload(idx, 4)[0])
        flat = idx.reshape(-1) >= 0
        assert torch.equal(planner.phy2log[a.reshape(-1)[flat]].long(), idx.reshape(-1)[flat])
        assert torch.equal(torch.bincount(a.reshape(-1)[flat]), torch.bincount(b.reshape(-1)[flat]))
    with pytest.raises(ValueError):
        planner.update_redundancy_mapping(torch.ones(n + 1, dtype=torch.int64, device="cuda"))


def test_the_tables_are_ready_on_every_stream():
    hist = torch.randperm(32, generator=torch.Generator().manual_seed(3))
    want = build_mapping(cube(), 1, 4, 1, hist)
    planner = Planner(cube(), 32 + 16, 32, 8, device="cuda", n_nodes=1)
    hist = hist.cuda()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # the current stream is busy for a while
    planner.update_redundancy_mapping(hist)
    with torch.cuda.stream(torch.cuda.Stream()):  # where a program moves its weights
        got = [t.cpu() for t in vars(planner.mapping).values()]
    for a, b in zip(got, vars(want).values()):
        assert torch.equal(a, b)


@pytest.mark.parametrize("history", ["none", "device", "host", "float"])
def test_a_graph_capture_refuses_a_new_placement(history):
    planner = Planner(cube(), 32 + 16, 32, 8, device="cuda", n_nodes=1)
    kept = planner.phy2log
    before, version = kept.clone(), planner.placement_version()
    hist = {"none": None, "device": torch.arange(32, device="cuda"), "host": torch.arange(32),
            "float": torch.rand(32, device="cuda")}[history]
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="captur"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            planner.update_redundancy_mapping(hist)
    torch.cuda.synchronize()
    assert planner.phy2log is kept and torch.equal(kept, before) and planner.placement_version() == version
    planner.update_redundancy_mapping(hist)  # and works again outside


def test_groups_whose_loads_pass_2_53_are_placed_as_on_the_host():
    # The groups hold the same loads in different orders: which of them is the heaviest is decided by
    # the rounding of the sums alone, so by the order in which the host adds them.
    planner = Planner(cube(), 4 * 48, 4 * 32, 32, device="cuda", n_nodes=2)
    g = torch.Generator().manual_seed(0)
    for bits in (48, 49, 55, 62):  # 32 loads of 48 bits stay below 2^53, of 49 bits may pass it
        for sign in (1, -1):
            loads = sign * (torch.randint(2 ** (bits - 1), 2**bits, (32,), generator=g) | 1)
            hist = torch.cat([loads[torch.randperm(32, generator=g)] for _ in range(4)])
            want = build_mapping(cube(), 4, 4, 1, hist, n_nodes=2)
            for h in (hist, hist.cuda()):
                got = planner.update_redundancy_mapping(h)
                for a, b in zip(got, (want.phy2log, want.log2phy, want.logcnt)):
                    assert torch.equal(a.cpu(), b), (bits, sign)


@pytest.mark.parametrize("entry", [None, (0, 3, 1, 8), (1, 2, 0, 8), (0, 0, 0, -1), (1, 7, 1, -1)])
def test_tables_that_disagree_with_the_topology_are_refused(entry):
    planner = Planner(cube(), 32 + 16, 32, 8, device="cuda", n_nodes=1)
    kept, version = planner.phy2log, planner.placement_version()
    before = kept.clone()
    tables = [planner.r2o.clone(), planner.o2r.clone()]
    if entry is None:  # ranks within range, but not the inverse
        tables[1] = tables[1].roll(1, 0)
    else:  # one past the last rank, or in front of the first
        which, rank, d, value = entry
        tables[which][rank, d] = value
    planner._engine.set_topology(*tables)
    with pytest.raises(AssertionError, match="inverse topology"):
        planner.update_redundancy_mapping(torch.arange(32))
    assert planner.phy2log is kept and torch.equal(kept, before) and planner.placement_version() == version
    planner._engine.set_topology(planner.r2o, planner.o2r)
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = torch.arange(32, device="cuda").unsqueeze(1)
    assert torch.equal(before[planner.run(idx, avail).long()].long(), idx)  # the engine's tables are untouched
    planner.update_redundancy_mapping(torch.arange(32))


@pytest.mark.parametrize("ranks,ll", [(2, 40), (8, 5), (8, 32), (16, 7), (32, 16), (33, 3)])
def test_packing_in_rounds_places_like_one_item_after_the_other(ranks, ll):
    """Histories where few items of a round count (a pack far below the others takes several in a
    row), where all do, and where empty experts fill up what is left."""
    n = ranks * ll
    r2o = ring(ranks)
    planner = Planner(r2o, n + ranks, n, ranks, device="cuda", n_nodes=1)
    k = torch.arange(1, n + 1)
    zipf = (1e6 / k**1.2).long()
    some = (torch.arange(n) % 3 == 0).long() * (k % 7 + 1)  # two thirds empty
    giant = torch.ones(n, dtype=torch.long)
    giant[n // 2] = 10**9
    halves = (2.0 ** (40 - (k % 40))).long()
    for hist in (zipf, zipf.flip(0), some, giant, giant - 1, halves, k):
        want = build_mapping(r2o, 1, ll, 1, hist, n_nodes=1)
        got = planner.update_redundancy_mapping(hist.cuda())
        for a, b in zip(got, (want.phy2log, want.log2phy, want.logcnt)):
            assert torch.equal(a.cpu(), b)

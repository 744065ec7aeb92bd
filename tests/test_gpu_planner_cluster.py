"""The planner step in one thread-block cluster against the grid-wide kernel: the same shares, and the same number of
tokens on every physical expert, at the edges of slices, rounds, rows of counts and lists."""

import re
from pathlib import Path

import pytest
import torch

from lplb_b200 import Planner, topology

gpu = pytest.mark.gpu
CSRC = Path(__file__).resolve().parents[1] / "lplb_b200" / "csrc"


def test_the_cluster_kernel_waits_for_its_predecessor_first():
    text = re.sub(r"//[^\n]*", "", (CSRC / "planner_cluster.cuh").read_text())
    body = text[re.search(r"cluster_run_kernel\(", text).start() :]
    statements = [s.strip() for s in body[body.index("{") + 1 :].split(";")]
    statements = [s for s in statements if "__shared__" not in s]
    assert statements[0] == "wait_predecessors()"
    assert text.count("wait_predecessors") == 1  # both roles run behind it


def test_a_cta_that_gave_up_waits_for_its_messages_beyond_the_callers_budget():
    text = re.sub(r"//[^\n]*", "", (CSRC / "planner_cluster.cuh").read_text())
    for role in ("cluster_solver", "cluster_worker"):
        body = text[text.index(f"void {role}(") :]
        body = body[: body.index("\n}")]
        after = body[body.rindex("cluster_wait();") + len("cluster_wait();") :]
        assert "if (late) await_landing(" in after and "timeout_ns" not in after
    assert "timeout_ns" not in text[text.index("void await_landing(") :].split("}")[0]


def _planner(r2o, groups, ll, combined=1, **kw):
    g, d = r2o.shape
    ep = g * groups
    return Planner(r2o, ep * ll + ep * d * combined, ep * ll, ep, device="cuda", n_nodes=1, **kw)


def _indices(planner, n, dtype, seed, masked=0.1):
    gen = torch.Generator("cuda").manual_seed(seed)
    e = planner.n_logical_routed_experts
    skew = torch.rand(e, device="cuda", generator=gen) ** 3 + 1e-3
    idx = torch.multinomial(skew, max(n, 1), replacement=True, generator=gen)[:n]
    idx[torch.rand(n, device="cuda", generator=gen) < masked] = -1
    planner.update_redundancy_mapping(torch.bincount(idx + 1, minlength=e + 1)[1:])
    return idx.to(dtype)


def _counts(planner, ids):
    return torch.bincount(ids.reshape(-1).long() + 1, minlength=planner.n_routed_experts + 1)


def _check(planner, idx, cluster, in_place=False):
    """Two steps in a cluster (a cold and, with warm starts, a warm one) against two of the grid-wide kernel."""
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    for step in range(2):
        results = []
        for c in (0, cluster):
            if step == 0:
                planner.invalidate_warm_start()
            else:  # the same anchor on both sides
                planner.invalidate_warm_start()
                eng.run_fused(idx, avail, 16, False)
            buf = idx.clone()
            out = eng.run_fused(buf, avail, 16, False, buf if in_place else None, c)
            results.append((out, eng.last_probs().clone()))
        (want, shares), (got, got_shares) = results
        assert torch.equal(got_shares, shares)
        assert torch.equal(_counts(planner, got), _counts(planner, want))
        live = idx >= 0
        assert torch.equal(planner.phy2log[got[live].long()].long(), idx[live].long())
        assert bool((got[~live] == -1).all())
    assert planner.check_status().ok


@gpu
@pytest.mark.parametrize("r2o,groups,ll", [(topology.cube(), 1, 32), (topology.cube(), 4, 8), (topology.cube(), 5, 4), (topology.ring(5), 2, 7),
                                            (topology.hypercube(), 1, 16), (topology.torus(8, 4), 1, 8)])
def test_each_kernel_continues_from_the_iterates_it_saved_itself(r2o, groups, ll):
    """The same batches on two planners, one always grid-wide, the other always in a cluster."""
    grid, cluster = (_planner(r2o, groups, ll, warm_start=True) for _ in range(2))
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    gen = torch.Generator("cuda").manual_seed(ll)
    e = grid.n_logical_routed_experts
    popularity = torch.rand(e, device="cuda", generator=gen) ** 3 + 1e-3
    for p in (grid, cluster):
        p.update_redundancy_mapping((popularity * 1e6).long())
    warm = 0
    for step in range(14):
        if step == 7:  # another distribution: the saved iterates do not fit
            popularity = torch.rand(e, device="cuda", generator=gen) ** 3 + 1e-3
        if step == 11:
            for p in (grid, cluster):
                p.invalidate_warm_start()
        idx = torch.multinomial(popularity, 15000, replacement=True, generator=gen)
        grid._engine.run_fused(idx, avail, 16, False, None, 0)
        out = cluster._engine.run_fused(idx, avail, 16, False, None, 16)
        assert torch.equal(cluster._engine.last_probs(), grid._engine.last_probs())
        assert torch.equal(cluster._engine.warm_start_valid(), grid._engine.warm_start_valid())
        want = grid._engine.map_idx(idx, grid._engine.last_probs(), grid.count_workload(idx, 8)[1], 8)
        assert torch.equal(_counts(cluster, out), _counts(grid, want))
        iters = [p.check_status(clear=True)["lp_iters"] for p in (grid, cluster)]
        assert iters[0] == iters[1]
        warm += step > 0 and iters[1] <= 3
    assert warm  # warm starts were among them


# 512 threads and slices in rounds of them with groups of 8 ranks, 256 with larger ones
@gpu
@pytest.mark.parametrize("n", [0, 1, 3, 31, 511, 512, 513, 1024, 1537, 4095, 7681, 30721, 153600])
@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_batches_at_the_edges_of_slices_and_rounds(n, dtype):
    planner = _planner(topology.cube(), 1, 32)
    idx = _indices(planner, n, dtype, seed=n)
    for cluster in (2, 4, 8, 16):
        if n <= (cluster - 1) * 10240:
            _check(planner, idx, cluster, in_place=cluster == 4)


@gpu
@pytest.mark.parametrize("r2o,groups,ll,combined", [
    (topology.ring(3), 1, 9, 1),                       # 27 experts: a row that is no whole number of messages
    (topology.ring(5), 2, 7, 3),                       # fewer ranks than rows of the tile
    (topology.cube(), 4, 8, 2),                        # one group to each of half of the warps
    (topology.cube(), 5, 4, 1),                        # more than half of the warps solve: nobody is left to send
    (topology.cube(), 16, 8, 1),                       # two rounds, 1024 experts
    (topology.circulant(8, (1, 2, 5)), 1, 6, 2),       # every expert replicated
    (topology.circulant(7, (1, 2, 3, 6)), 3, 48, 1),   # 1008 experts
    (topology.hypercube(), 1, 16, 1), (topology.circulant(12, (1, 2, 5, 7)), 2, 5, 1),
    (topology.torus(8, 4), 1, 32, 1), (topology.circulant(20, (1, 7, 9)), 1, 3, 1),
])
@pytest.mark.parametrize("warm", [True, False])
def test_every_shape_of_groups(r2o, groups, ll, combined, warm):
    planner = _planner(r2o, groups, ll, combined, warm_start=warm)
    for n, cluster in ((700, 2), (1025 * 8, 16)):
        _check(planner, _indices(planner, n, torch.int64, seed=ll), cluster)


@gpu
def test_shapes_and_batches_that_do_not_fit_take_the_grid_wide_kernel():
    for r2o, groups, ll, n in ((topology.cube(), 1, 32, 153601), (topology.cube(), 17, 8, 4096), (topology.ring(8), 1, 200, 4096),
                               (topology.torus(8, 4), 1, 8, 15361), (topology.torus(8, 8), 1, 8, 2000), (topology.ring(80), 1, 4, 2000)):
        planner = _planner(r2o, groups, ll)
        idx = _indices(planner, n, torch.int64, seed=1)
        avail = torch.zeros(1, dtype=torch.int32, device="cuda")
        with pytest.raises(RuntimeError):
            planner._engine.run_fused(idx, avail, 16, False, None, 16)
        out = planner.run(idx, avail)
        assert int(avail) == groups
        staged = planner._engine.map_idx(idx, planner.last_probs.contiguous(), planner.count_workload(idx, 8)[1], 8)
        assert torch.equal(_counts(planner, out), _counts(planner, staged))


@gpu
def test_bad_indices_are_counted_and_masked():
    planner = _planner(topology.cube(), 1, 8)
    idx = _indices(planner, 2000, torch.int64, seed=4, masked=0.0)
    idx[::10] = 64
    idx[1::10] = -7
    idx[2::10] = (1 << 32) + 5  # in range if its upper half were lost
    out = planner._engine.run_fused(idx, torch.zeros(1, dtype=torch.int32, device="cuda"), 16, False, None, 8)
    bad = (idx < 0) | (idx >= 64)
    assert bool((out[bad] == -1).all()) and bool((out[~bad] >= 0).all())
    st = planner.check_status(clear=True)
    assert st["bad_indices"] == int(bad.sum()) and st["error"] == "bad_index"


@gpu
def test_clusters_and_grids_alternate_on_one_engine_without_a_gap():
    planner = _planner(topology.cube(), 1, 16)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    batches = [_indices(planner, n, torch.int64, seed=n) for n in (100, 20000, 3000)]
    outs = []
    before = eng.completed_launches()
    for i in range(30):  # each step's indices come from a kernel right in front of it
        idx = batches[i % 3].clone()
        outs.append((idx, eng.run_fused(idx, avail, 16, False, None, (0, 4, 16)[i * 7 % 3]), eng.last_probs().clone()))
    assert eng.completed_launches() == before + 30 and int(avail) == 30 and planner.check_status().ok
    for idx, out, shares in outs:
        want = eng.map_idx(idx, shares, planner.count_workload(idx, 8)[1], 8)
        assert torch.equal(_counts(planner, out), _counts(planner, want))


@gpu
def test_the_exchange_runs_in_a_cluster_too():
    planner = _planner(topology.cube(), 1, 8, peer_timeout_us=300.0)
    eng = planner._engine
    eng.open_exchange_loopback(2, 0)
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    peer = torch.arange(64, dtype=torch.int32) * 3
    for step in range(3):
        idx = _indices(planner, 4096, torch.int64, seed=step)
        eng.debug_fill_slot(1, peer, eng.completed_launches() + 1)
        out = eng.run_fused(idx, avail, 16, True, None, (2, 8, 16)[step])
        assert planner.check_status().ok
        counts = torch.bincount(idx + 1, minlength=65)[1:].int()
        glob = eng.workspace()[8 + 2 * 64 : 8 + 3 * 64]
        assert torch.equal(glob.cpu(), counts.cpu() + peer)
        want = eng.map_idx(idx, eng.last_probs(), planner.count_workload(idx, 8)[1], 8)
        assert torch.equal(_counts(planner, out), _counts(planner, want))
    # a peer that never publishes: reported, solved from this rank's counts, nothing kept for a warm start
    idx = _indices(planner, 4096, torch.int64, seed=9)
    eng.run_fused(idx, avail, 16, True, None, 8)
    st = planner.check_status(clear=True)
    assert st["error"] == "peer_timeout" and st["detail"] == 0b10 and st["timeouts"] == 1
    assert int(eng.warm_start_valid().sum()) == 0


def _clean_step(planner, idx, use_exchange=False, cluster=8):
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = eng.run_fused(idx, avail, 16, use_exchange, None, cluster)
    want = eng.map_idx(idx, eng.last_probs(), planner.count_workload(idx, 8)[1], 8)
    assert torch.equal(_counts(planner, out), _counts(planner, want)) and planner.check_status().ok


@gpu
@pytest.mark.parametrize("cluster", [2, 4, 16])
def test_workers_whose_wait_runs_out_leave_half_of_the_tokens(cluster):
    """The solver still waits for a peer that never publishes when the workers give up."""
    planner = _planner(topology.cube(), 1, 8, peer_timeout_us=3000.0, grid_timeout_us=300.0)
    eng = planner._engine
    eng.open_exchange_loopback(2, 0)
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = _indices(planner, 6000, torch.int64, seed=11)
    out = eng.run_fused(idx, avail, 16, True, None, cluster)
    st = planner.check_status(clear=True)
    assert st["error"] == "lp_timeout" and st["timeouts"] == cluster  # every worker, and the missing peer
    live = idx >= 0
    assert torch.equal(planner.phy2log[out[live].long()].long(), idx[live]) and bool((out[~live] == -1).all())
    replicated = planner.mapping.log2phy[:, 1] >= 0
    moved = torch.bincount(idx[live & (out == planner.mapping.log2phy[idx.clamp_min(0), 1])], minlength=64)
    counts = torch.bincount(idx[live], minlength=64)
    assert bool((moved[~replicated] == 0).all())
    # every other one of a worker's tokens, the first of them
    assert bool((moved[replicated] >= counts[replicated] // 2).all())
    assert bool((moved[replicated] <= (counts[replicated] + cluster - 1) // 2).all())
    eng.debug_fill_slot(1, torch.zeros(64, dtype=torch.int32), eng.completed_launches() + 1)
    _clean_step(planner, idx, use_exchange=True)


@gpu
@pytest.mark.parametrize("cluster", [2, 16])
def test_a_solver_whose_wait_runs_out_reports_it(cluster):
    planner = _planner(topology.cube(), 1, 32)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = _indices(planner, 10240 * (cluster - 1), torch.int64, seed=cluster)
    eng.set_params(24, 1e-4, 1e6, 1e-3)  # the ids come over PCIe, so no count is there within a nanosecond
    for _ in range(3):
        out = eng.run_fused(idx.cpu().pin_memory(), avail, 16, False, torch.empty_like(idx), cluster)
        st = planner.check_status(clear=True)
        assert st["error"] in ("grid_timeout", "lp_timeout") and st["timeouts"] >= 1
        live = idx >= 0
        assert torch.equal(planner.phy2log[out[live].long()].long(), idx[live]) and bool((out[~live] == -1).all())
    eng.set_params(24, 1e-4, 1e6, 1e6)
    _clean_step(planner, idx, cluster=16)


def test_the_rows_of_counts_are_cleared_before_a_worker_may_write_them():
    text = re.sub(r"//[^\n]*", "", (CSRC / "planner_cluster.cuh").read_text())
    body = text[text.index("void cluster_solver(") :]
    assert "reinterpret_cast<int4*>(rows)[i] = int4{0, 0, 0, 0}" in body[: body.index("cluster_arrive();")]


@gpu
def test_counts_that_came_late_are_a_part_of_the_batch():
    """Every batch is drawn from experts of its own, so whatever else lies in shared memory shows up as a token too many."""
    planner = _planner(topology.cube(), 1, 32)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    gen = torch.Generator("cuda").manual_seed(2)
    for step in range(24):
        own = torch.arange(256, device="cuda")[step % 8 :: 8]
        idx = own[torch.randint(32, (150000,), device="cuda", generator=gen)]
        eng.set_params(24, 1e-4, 1e6, 1e6 if step % 2 == 0 else 1e-3)
        src = idx if step % 2 == 0 else idx.cpu().pin_memory()
        eng.run_fused(src, avail, 16, False, torch.empty_like(idx), 16)
        counts = torch.bincount(idx, minlength=256)
        glob = eng.workspace()[8 + 2 * 256 : 8 + 3 * 256]
        assert bool((glob >= 0).all()) and bool((glob <= counts).all())
        st = planner.check_status(clear=True)
        assert st.ok == (step % 2 == 0)
        assert not st.ok or torch.equal(glob.long(), counts)


def test_whichever_thread_gives_up_reports_it():
    text = re.sub(r"//[^\n]*", "", (CSRC / "planner_cluster.cuh").read_text())
    assert not re.search(r"late && threadIdx|threadIdx\.x == 0 && late", text)
    for role, code in (("cluster_solver", "kErrGridTimeout"), ("cluster_worker", "kErrLpTimeout")):
        body = text[text.index(f"void {role}(") :]
        assert re.search(rf"\n *report_late\(late, reported, status, {code}", body[: body.index("\n}")])


@gpu
@pytest.mark.parametrize("cluster", [2, 16])
def test_a_step_without_a_report_had_all_counts(cluster):
    """Budgets around the time at which the counts arrive (the ids come over PCIe): some warps give up on them, others
    still see them."""
    planner = _planner(topology.cube(), 1, 32)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = _indices(planner, 10240 * (cluster - 1), torch.int64, seed=21)
    host, out = idx.cpu().pin_memory(), torch.empty_like(idx)
    counts = torch.bincount(idx + 1, minlength=257)[1:]
    by_cta = planner.count_workload(idx, 8)[1]
    reported = 0
    for step in range(250):
        eng.set_params(24, 1e-4, 1e6, 0.001 + 0.2 * step)
        eng.run_fused(host, avail, 16, False, out, cluster)
        glob = eng.workspace()[8 + 2 * 256 : 8 + 3 * 256].clone()
        st = planner.check_status(clear=True)
        reported += not st.ok
        if st.ok:
            assert torch.equal(glob.long(), counts)
            want = eng.map_idx(idx, eng.last_probs(), by_cta, 8)
            assert torch.equal(_counts(planner, out), _counts(planner, want))
    assert 0 < reported < 250


@gpu
@pytest.mark.parametrize("r2o,ll", [(topology.cube(), 32), (topology.hypercube(), 16), (topology.torus(8, 4), 8)])
@pytest.mark.parametrize("n", [8, 4096, 15360, 15368, 32768])
def test_a_result_in_host_memory_takes_the_cluster_for_small_batches_only(r2o, ll, n):
    planner = _planner(r2o, 1, ll)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = _indices(planner, n, torch.int64, seed=n).reshape(-1, 8)
    by_cta = planner.count_workload(idx, 8)[1]
    host = idx.cpu().pin_memory()
    assert (eng.cluster_choice(n, host_result=True) > 0) == (n <= 15360)
    for src, out in ((host, None), (host, torch.empty_like(idx)), (idx, torch.empty_like(host).pin_memory())):
        got = planner.run(src, avail, out=out)
        torch.cuda.synchronize()
        assert got.is_cuda == (out is not None and out.is_cuda)
        want = eng.map_idx(idx, eng.last_probs(), by_cta, 8)
        assert torch.equal(_counts(planner, got.cuda()), _counts(planner, want))
        assert torch.equal(planner.phy2log[got.cuda()[idx >= 0]].long(), idx[idx >= 0])
    assert planner.check_status().ok


@gpu
@pytest.mark.parametrize("r2o,groups,ll", [(topology.torus(8, 8), 1, 2), (topology.cube(), 17, 2), (topology.cube(), 1, 150), (topology.ring(80), 1, 2),
                                            (topology.cube(), 1, 2), (topology.hypercube(), 1, 2), (topology.torus(8, 4), 1, 2)])
def test_an_empty_batch_runs_on_every_shape(r2o, groups, ll):
    planner = _planner(r2o, groups, ll)
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = planner.run(torch.zeros(0, 8, dtype=torch.int64, device="cuda"), avail)
    assert out.shape == (0, 8) and int(avail) == groups and planner.check_status().ok
    assert bool((planner.last_probs == 1).all())


@gpu
@pytest.mark.parametrize("r2o,groups,ll,combined,most", [
    (topology.cube(), 1, 64, 1, 153600), (topology.cube(), 1, 32, 1, 122880), (topology.cube(), 1, 32, 2, 92160), (topology.cube(), 2, 16, 1, 92160),
    (topology.cube(), 4, 8, 1, 61440), (topology.ring(3), 1, 9, 1, 92160), (topology.cube(), 4, 8, 2, 30720), (topology.circulant(8, (1, 2, 5)), 1, 6, 2, 30720),
    (topology.hypercube(), 1, 4, 2, 38400), (topology.torus(8, 4), 1, 8, 1, 15360), (topology.torus(8, 8), 1, 8, 1, 0), (topology.cube(), 17, 8, 1, 0),
])
@pytest.mark.parametrize("is64", [True, False])
def test_the_largest_batch_of_a_cluster_follows_the_share_of_replicated_experts(r2o, groups, ll, combined, most, is64):
    eng = _planner(r2o, groups, ll, combined)._engine
    assert eng.cluster_choice(0, is64) == (2 if most else 0)
    assert eng.cluster_choice(most + 1, is64) == 0
    if most:
        assert eng.cluster_choice(most, is64) == 16 and eng.cluster_choice(256, is64) == 2 and eng.cluster_choice(257, is64) == 4


# 224 threads take the totals two at a time while one warp rehearses, 256 one at a time where none does (five groups)
@gpu
@pytest.mark.parametrize("groups,ll", [(1, 27), (1, 28), (1, 29), (1, 32), (1, 56), (1, 57), (4, 14), (1, 112), (1, 113), (1, 200), (5, 8), (5, 13)])
@pytest.mark.parametrize("r2o", [topology.ring(8), topology.circulant(8, (1, 2, 5))])
def test_the_grid_wide_step_at_the_edges_of_its_rounds_of_experts(r2o, groups, ll):
    planner = _planner(r2o, groups, ll, warm_start=False)
    eng = planner._engine
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    for n in (500, 20000):
        idx = _indices(planner, n, torch.int64, seed=n + ll)
        out = eng.run_fused(idx, avail, 16, False, None, 0)
        counts, by_cta = planner.count_workload(idx, 8)
        shares = eng.last_probs().clone()
        glob = eng.workspace()[8 + 2 * counts.numel() : 8 + 3 * counts.numel()]
        assert torch.equal(glob, counts)
        assert torch.equal(shares, planner.solve_probs(counts, avail)[0])
        assert torch.equal(_counts(planner, out), _counts(planner, eng.map_idx(idx, shares, by_cta, 8)))
    assert planner.check_status().ok


@gpu
def test_an_engine_without_replicas_takes_the_grid_wide_kernel():
    """The planner refuses such a placement, the engine does not; a cluster's messages are one per replicated expert."""
    from lplb_b200 import _native

    eng = _native.load().PlannerEngine(1, 8, 2, 4, 0, 0)
    eng.set_topology(topology.cube(), topology.invert_r2o(topology.cube()))
    ids = torch.arange(32, device="cuda")
    eng.set_mapping(ids, torch.stack([ids, torch.full_like(ids, -1)], 1).contiguous(), torch.full_like(ids, -1))
    avail = torch.zeros(1, dtype=torch.int32, device="cuda")
    idx = torch.arange(-1, 1000, device="cuda") % 33 - 1
    with pytest.raises(RuntimeError):
        eng.run_fused(idx, avail, 16, False, None, 2)
    assert eng.cluster_choice(idx.numel()) == 0
    assert torch.equal(eng.run_fused(idx, avail, 16, False, None, -1), idx)

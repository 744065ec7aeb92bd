"""Performance cases of the framework: what a training or serving program has it do.

Four kinds of work, all through the public entry points:

* ``run``      ``Planner.run``: a batch of logical expert ids in, physical ids out (every batch)
* ``solve``    ``Planner.solve_probs``: shares from statistics that the caller gathered itself
* ``replace``  ``Planner.update_redundancy_mapping``: a new expert placement (every N steps)
* ``moe``      ``MoELayer.forward``: routing by the per-batch LP, dispatch, both grouped GEMMs, combine

``prepare`` makes what such a program holds (a planner or a layer, a few consecutive batches of
one routing distribution), ``run`` is one call on the next of these batches.
"""

import torch

from lplb_b200 import Planner, topology
from lplb_b200.models.moe import MoELayer

N_BATCHES = 3  # consecutive batches held per state


def listed():
    return [
        # decode step of a serving program, captured once in a CUDA graph and replayed: 128 tokens
        # per rank is the smallest batch of the torus sweep
        dict(name="run_decode_graph", kind="run", topology="cube", groups=1, local_logical=32, combined=1, tokens=128,
             topk=8, int32=False, padded=False, graph=True),
        # the headline workload: EP8 Cube, 256 + 16 experts, 4096 tokens x top-8
        dict(name="run_cube", kind="run", topology="cube", groups=1, local_logical=32, combined=1, tokens=4096, topk=8,
             int32=False, padded=False, graph=False),
        # the largest batch of the torus sweep (64 experts per rank), int32 ids from a custom gate
        dict(name="run_torus_large", kind="run", topology="torus2x4", groups=1, local_logical=64, combined=1,
             tokens=16384, topk=8, int32=True, padded=False, graph=False),
        # EP32 training: four LP groups of a cube, a ragged batch with masked-out (-1) entries
        dict(name="run_ep32_ragged", kind="run", topology="cube", groups=4, local_logical=8, combined=1, tokens=1025,
             topk=8, int32=False, padded=True, graph=False),
        # EP32 on one 8x4 torus: a 32-rank LP group, in a captured graph
        dict(name="run_torus8x4_graph", kind="run", topology="torus8x4", groups=1, local_logical=8, combined=1,
             tokens=4096, topk=8, int32=False, padded=False, graph=True),
        # offline evaluation of 64 unrelated Cube instances per call (the solver microbenchmark)
        dict(name="solve_cube_batch", kind="solve", topology="cube", groups=64, local_logical=16, warm=False),
        # one 64-rank group whose statistics the caller accumulated itself
        dict(name="solve_torus8x8", kind="solve", topology="torus8x8", groups=1, local_logical=8, warm=False),
        # re-placement from the load history (the balancer, every table, upload to the device)
        dict(name="replace_cube", kind="replace", topology="cube", groups=1, local_logical=32, combined=1),
        # the MoE layer in decode (weights bound), at a ragged middle size, with the dispatch fused
        # into the first GEMM, and at the full batch of the layer benchmark (tensor bound)
        dict(name="moe_decode", kind="moe", topology="cube", local_logical=4, hidden=7168, inter=2048, topk=8,
             tokens=64, fused=False),
        dict(name="moe_ragged", kind="moe", topology="cube", local_logical=4, hidden=7168, inter=2048, topk=8,
             tokens=1000, fused=False),
        dict(name="moe_fused", kind="moe", topology="cube", local_logical=4, hidden=7168, inter=2048, topk=8,
             tokens=4096, fused=True),
        dict(name="moe_full", kind="moe", topology="cube", local_logical=4, hidden=7168, inter=2048, topk=8,
             tokens=8192, fused=False),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "solve", "solve", "replace", "moe", "moe", "moe"])
    if kind == "moe":
        return dict(kind="moe", topology=rng.choice(["cube", "ring8"]), local_logical=rng.randint(2, 8),
                    hidden=256 * rng.randint(4, 28), inter=128 * rng.randint(2, 16), topk=rng.choice([1, 2, 4, 6, 8]),
                    tokens=_log_uniform(rng, 16, 8192), fused=rng.random() < 0.3)
    if kind == "solve":
        name = rng.choice(["ring8", "cube", "torus2x4", "hypercube", "torus8x4", "torus8x8"])
        ranks = int(topology.by_name(name).shape[0])
        return dict(kind="solve", topology=name, groups=_log_uniform(rng, 1, 512 // ranks),
                    local_logical=rng.randint(4, 16), warm=rng.random() < 0.5)
    name = rng.choice(["cube", "cube", "torus2x4", "ring8", "hypercube", "torus8x4"])
    ranks = int(topology.by_name(name).shape[0])
    groups = rng.choice([1, 2, 4]) if ranks == 8 else 1
    local_logical = rng.randint(8, 512 // (ranks * groups))
    combined = rng.choice([1, 1, 2])
    if kind == "replace":
        return dict(kind="replace", topology=name, groups=groups, local_logical=local_logical, combined=combined)
    return dict(kind="run", topology=name, groups=groups, local_logical=local_logical, combined=combined,
                tokens=_log_uniform(rng, 32, 16384), topk=rng.choice([1, 2, 4, 6, 8]), int32=rng.random() < 0.3,
                padded=rng.random() < 0.3, graph=rng.random() < 0.4)


def _shape(case):
    ranks, dup = (int(v) for v in topology.by_name(case["topology"]).shape)
    ep = ranks * case.get("groups", 1)
    n_logical = ep * case["local_logical"]
    return ranks, dup, ep, n_logical, n_logical + ep * dup * case.get("combined", 1)


def _planner(case, **kw):
    _, _, ep, n_logical, n_physical = _shape(case)
    return Planner(topology.by_name(case["topology"]), n_physical, n_logical, ep, device="cuda", n_nodes=1, **kw)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _gate(g, tokens, n_logical, topk, bias):
    """Top-k of bf16 logits ~ N(0, 1) plus a per-expert bias, as the headline benchmark draws them."""
    logits = torch.randn(tokens, n_logical, device="cuda", generator=g) + bias
    return torch.softmax(logits.bfloat16().float(), -1).topk(topk, dim=-1)


def prepare(case, seed):
    return {"run": _prepare_run, "solve": _prepare_solve, "replace": _prepare_replace, "moe": _prepare_moe}[case["kind"]](
        case, seed
    )


def run(state):
    return state["pass"](state)


def _next(state):
    state["step"] += 1
    return state["batches"][state["step"] % N_BATCHES]


# ---------------------------------------------------------------------------------------- run
def _prepare_run(case, seed):
    g = _generator(seed)
    n_logical = _shape(case)[3]
    bias = torch.randn(n_logical, device="cuda", generator=g)
    batches = []
    for _ in range(N_BATCHES):
        idx = _gate(g, case["tokens"], n_logical, case["topk"], bias).indices
        if case["padded"]:  # tokens past the end of a sequence
            idx = torch.where(torch.rand(idx.shape, device="cuda", generator=g) < 0.06, torch.full_like(idx, -1), idx)
        batches.append(idx.int() if case["int32"] else idx)
    planner = _planner(case)
    history = torch.bincount(torch.cat(batches).reshape(-1).long() + 1, minlength=n_logical + 1)[1:]
    planner.update_redundancy_mapping(history)
    state = {
        "planner": planner, "batches": batches, "step": 0, "pass": _pass_run,
        "avail": torch.zeros(1, dtype=torch.int32, device="cuda"),
        # expert behind every physical slot, with -1 behind the masked entries
        "expert_of": torch.cat([planner.phy2log, planner.phy2log.new_full((1,), -1)]),
    }
    if case["graph"]:
        state["idx"], state["out"] = batches[0].clone(), torch.empty_like(batches[0])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _step_run(state, state["idx"], state["out"])
        torch.cuda.current_stream().wait_stream(side)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["result"] = _step_run(state, state["idx"], state["out"])
        state["pass"] = _pass_run_graph
    return state


def _step_run(state, idx, out=None):
    # Which of an expert's tokens go to its replica is free (only how many is fixed), so the ids are
    # taken on to the expert whose weights they select, beside the shares that fix the split.
    phys = state["planner"].run(idx, state["avail"], out=out)
    return {"expert": state["expert_of"][phys], "shares": state["planner"].last_probs, "solved": state["avail"]}


def _pass_run(state):
    return _step_run(state, _next(state))


def _pass_run_graph(state):
    state["idx"].copy_(_next(state))
    state["graph"].replay()
    return state["result"]


# -------------------------------------------------------------------------------------- solve
def _prepare_solve(case, seed):
    g = _generator(seed)
    n_logical = _shape(case)[3]
    ll = case["local_logical"]

    def popularity():  # Dirichlet(0.3) expert popularity, as the solver microbenchmark draws it
        alpha = torch.full((n_logical // ll, ll), 0.3, device="cuda")
        p = torch._standard_gamma(alpha, generator=g)
        return (p / p.sum()).sort(dim=-1, descending=True).values.reshape(-1)  # heaviest experts are the replicated ones

    base = popularity()
    batches = []
    for _ in range(N_BATCHES):
        # warm: consecutive batches of one distribution; cold: unrelated instances
        p = base * (1 + 0.05 * torch.randn(n_logical, device="cuda", generator=g)).clamp_min(0) if case["warm"] else popularity()
        batches.append((p * (32768 * n_logical / 16)).int())
    return {"planner": _planner(case, warm_start=case["warm"]), "batches": batches, "step": 0, "pass": _pass_solve,
            "avail": torch.zeros(1, dtype=torch.int32, device="cuda")}


def _pass_solve(state):
    shares, normalised = state["planner"].solve_probs(_next(state), state["avail"])
    return {"shares": shares, "normalised": normalised, "solved": state["avail"]}


# ------------------------------------------------------------------------------------ replace
def _prepare_replace(case, seed):
    g = _generator(seed)
    n_logical = _shape(case)[3]
    popularity = torch.softmax(torch.randn(n_logical, device="cuda", generator=g), -1)
    batches = [(popularity * (1 + 0.2 * torch.rand(n_logical, device="cuda", generator=g)) * 1e7).long() for _ in range(N_BATCHES)]
    return {"planner": _planner(case), "batches": batches, "step": 0, "pass": _pass_replace}


def _pass_replace(state):
    return list(state["planner"].update_redundancy_mapping(_next(state)))


# ---------------------------------------------------------------------------------------- moe
def _prepare_moe(case, seed):
    g = _generator(seed)
    n_logical = _shape(case)[3]
    bias = 0.5 * torch.randn(n_logical, device="cuda", generator=g)
    batches = []
    for _ in range(N_BATCHES):
        x = torch.randn(case["tokens"], case["hidden"], device="cuda", generator=g).bfloat16()
        weights, idx = _gate(g, case["tokens"], n_logical, case["topk"], bias)
        batches.append((x, idx, weights))
    planner = _planner(case)
    planner.update_redundancy_mapping(torch.bincount(torch.cat([b[1] for b in batches]).reshape(-1), minlength=n_logical))
    layer = MoELayer(planner, case["hidden"], case["inter"], case["topk"], max_tokens=case["tokens"], seed=seed)
    layer.fuse_dispatch = case["fused"]
    return {"layer": layer, "batches": batches, "step": 0, "pass": _pass_moe,
            "avail": torch.zeros(1, dtype=torch.int32, device="cuda")}


def _pass_moe(state):
    x, idx, weights = _next(state)
    return {"y": state["layer"].forward(x, idx, weights, state["avail"]), "solved": state["avail"]}


# --------------------------------------------------------------------------------------- work
def work(case):
    ranks, dup, ep, n_logical, n_physical = _shape(case)
    # about four interior-point iterations from scratch, two from a saved iterate: one ranks^3 / 3
    # factorisation and three pairs of triangular solves each, in float64
    per_iteration = ep // ranks * (2 * ranks**3 / 3 + 6 * ranks**2 * 2)
    if case["kind"] == "solve":
        return {"bytes": 4 * (2 * n_logical + ep * dup), "flops": (2 if case["warm"] else 4) * per_iteration}
    if case["kind"] == "replace":
        return {"bytes": 8 * n_logical + 4 * (n_physical + 3 * n_logical), "flops": 0}
    ids = case["tokens"] * case["topk"] * (4 if case.get("int32") else 8)
    if case["kind"] == "run":
        return {"bytes": 2 * ids + 4 * case["tokens"] * case["topk"] + 4 * (3 * n_logical + ep * dup),
                "flops": 2 * per_iteration}
    pairs = case["tokens"] * case["topk"]
    per_expert = 3 * case["hidden"] * case["inter"]
    touched = n_physical * (1 - (1 - 1 / n_physical) ** pairs)  # experts that at least one pair reaches
    return {"bytes": 2 * per_expert * touched + 2 * 2 * case["tokens"] * case["hidden"] + ids,
            "flops": 2 * per_expert * pairs}


def tolerance(case):
    if case["kind"] == "replace":
        return "exact"
    if case["kind"] == "moe":
        # bf16 activations between the GEMMs and bf16 rows before the weighted sum: against the same
        # layer in fp32 1.4e-3 and, at the worst element, 0.018
        return {"rel": 6e-3, "max": 0.08}
    # float32 shares of a float64 iteration that walks the same iterates in any order of its sums
    # (warp against thread-block solver: 1e-11 at most); one float32 unit here and there is left
    return {"rel": 1e-5, "max": 1e-4}

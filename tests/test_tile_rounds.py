"""Tile solver with eight tile rows: pivots that the topology leaves uncoupled go in one round (device code on the CPU)."""

import pytest
import torch
from test_sim_solver import _solve_tiles, sim  # noqa: F401

from lplb_b200 import lp, topology


def _within_blocks(g):
    """Edges inside every block of eight ranks only: no tile row is coupled to another."""
    return torch.tensor([[i // 8 * 8 + (i % 8 + s) % min(8, g - i // 8 * 8) for s in (1, 3)] for i in range(g)], dtype=torch.int32)


def _random(g, d, seed):
    gen = torch.Generator().manual_seed(seed)
    cols = []
    while len(cols) < d:
        p = torch.randperm(g, generator=gen)
        if not bool((p == torch.arange(g)).any()):
            cols.append(p)
    return torch.stack(cols, 1).int()


@pytest.mark.parametrize("name,r2o", [
    ("a ring of tile rows, four rounds", topology.torus(8, 8)),
    ("a ring with a last row of one rank", topology.circulant(41, (1, 8))),
    ("one replica", topology.ring(64)),
    ("no coupling, one round", _within_blocks(64)),
    ("no coupling, a last row of three ranks", _within_blocks(51)),
    ("two rings of four rows", torch.cat([topology.torus(4, 8), topology.torus(4, 8) + 32])),
    ("every row with every other, eight rounds", topology.circulant(64, (8, 16, 24, 32))),
    ("random", _random(57, 3, 1)), ("random, sparse", _random(64, 1, 2)),
])
def test_pivots_in_rounds_solve_like_one_after_the_other(sim, name, r2o):  # noqa: F811
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(5)
    cnt = ((torch.randn(1, g, 8, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
    f, iters, conv = _solve_tiles(sim, r2o, w, fixed)
    ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4)
    assert conv.all() and iters.tolist() == ref.iters.tolist()
    assert float((f - ref.f).abs().max()) < 1e-5  # as for the other sizes: the step lengths carry 26 bits

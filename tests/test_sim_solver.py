"""Run the CUDA solver's device code on the CPU through the lock-step warp emulation
(csrc/host_sim.h) and compare it with the float64 oracle."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

from lplb_b200 import lp, topology

CSRC = Path(__file__).resolve().parents[1] / "lplb_b200" / "csrc"


@pytest.fixture(scope="module")
def sim(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    so = tmp_path_factory.mktemp("sim") / "libsim.so"
    subprocess.run(
        ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", str(CSRC / "sim_solver.cpp"), "-o", str(so)],
        check=True,
    )
    return ctypes.CDLL(str(so))


def _solve(lib, r2o, w, fixed, max_iters=24, tol=1e-4):
    g, d = r2o.shape
    nb = w.shape[0]
    r = np.ascontiguousarray(r2o.numpy().astype(np.int32))
    o = np.ascontiguousarray(topology.invert_r2o(r2o).numpy().astype(np.int32))
    wa = np.ascontiguousarray(w.numpy().astype(np.float64))
    fa = np.ascontiguousarray(fixed.numpy().astype(np.float64))
    f = np.zeros((nb, g, d))
    iters = np.zeros(nb, np.int32)
    conv = np.zeros(nb, np.int32)
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    rc = lib.lplb_sim_solve(g, d, ptr(r), ptr(o), nb, ptr(wa), ptr(fa), max_iters, ctypes.c_double(tol), ptr(f), ptr(iters), ptr(conv))
    assert rc == 0
    return torch.from_numpy(f), iters, conv


@pytest.mark.parametrize("name,nb", [("cube", 9), ("ring8", 6), ("hypercube", 3), ("ring5", 5), ("torus2x4", 4)])
def test_device_solver_matches_oracle(sim, name, nb):
    r2o = topology.by_name(name)
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(7)
    cnt = ((torch.randn(nb, g, 8, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
    if nb > 2:  # an empty group sharing a warp with live ones
        w[2], fixed[2] = 0, 0
    f, iters, conv = _solve(sim, r2o, w, fixed)
    assert conv.all() and bool(((f >= 0) & (f <= 1)).all())
    for i in range(nb):
        if float(w[i].sum() + fixed[i].sum()) == 0:
            assert torch.equal(f[i], torch.ones(g, d, dtype=torch.float64)) and iters[i] == 0
            continue
        _, t_opt = lp.solve_highs(w[i], fixed[i], r2o)
        mine = float(lp.rank_loads(f[i], w[i], fixed[i], r2o).max())
        assert -1e-9 < (mine - t_opt) / t_opt < 1e-3
        assert 1 <= iters[i] <= 12


def test_device_solver_follows_the_torch_restatement(sim):
    r2o = topology.cube()
    gen = torch.Generator().manual_seed(3)
    cnt = ((torch.randn(8, 8, 8, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :2].contiguous(), cnt[:, :, 2:].sum(-1)
    f, iters, _ = _solve(sim, r2o, w, fixed)
    ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4)
    assert iters.tolist() == ref.iters.tolist()
    assert float((f - ref.f).abs().max()) < 1e-5


def test_iteration_cap_is_reported(sim):
    r2o = topology.cube()
    w = torch.rand(2, 8, 2, dtype=torch.float64, generator=torch.Generator().manual_seed(1)) * 1000
    fixed = torch.rand(2, 8, dtype=torch.float64, generator=torch.Generator().manual_seed(2)) * 1000
    f, iters, conv = _solve(sim, r2o, w, fixed, max_iters=1, tol=1e-9)
    assert not conv.any() and iters.tolist() == [1, 1]
    assert bool(((f >= 0) & (f <= 1)).all())


def test_warm_start_on_device_code_matches_the_torch_restatement(sim):
    """A stream of similar batches, then a shifted one: the anchor logic of the device code
    (run under warp emulation) takes the same decisions and iterations as lp.solve_ipm."""
    r2o = topology.cube()
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(11)
    mean = (torch.rand(g, 8, generator=gen, dtype=torch.float64) + 0.5) * 4096
    anchor_c = np.zeros((1, g, 4 * d + 3))
    valid_c = np.zeros(1, np.int32)
    anchor_t = None
    r = np.ascontiguousarray(r2o.numpy().astype(np.int32))
    o = np.ascontiguousarray(topology.invert_r2o(r2o).numpy().astype(np.int32))
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    seen = []
    for step in range(5):
        if step == 3:
            mean = mean.flip(0) * torch.linspace(0.3, 2.0, 8, dtype=torch.float64)  # the distribution moves
        cnt = (mean * (1 + 0.02 * torch.randn(g, 8, generator=gen, dtype=torch.float64))).floor().unsqueeze(0)
        w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
        ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4, warm_start=True, anchor=anchor_t)
        anchor_t = ref.anchor
        wa, fa = np.ascontiguousarray(w.numpy()), np.ascontiguousarray(fixed.numpy())
        f = np.zeros((1, g, d))
        iters, conv = np.zeros(1, np.int32), np.zeros(1, np.int32)
        rc = sim.lplb_sim_solve_warm(g, d, ptr(r), ptr(o), 1, ptr(wa), ptr(fa), 24, ctypes.c_double(1e-4), ptr(f),
                                     ptr(iters), ptr(conv), ptr(anchor_c), ptr(valid_c), ctypes.c_double(0.05),
                                     ctypes.c_double(1e-3))
        assert rc == 0 and conv[0] == 1
        assert int(iters[0]) == int(ref.iters[0])
        assert float((torch.from_numpy(f) - ref.f).abs().max()) < 1e-5
        _, t_opt = lp.solve_highs(w[0], fixed[0], r2o)
        assert (float(lp.rank_loads(torch.from_numpy(f[0]), w[0], fixed[0], r2o).max()) - t_opt) / t_opt < 1e-3
        seen.append((bool(ref.warm[0]), int(iters[0])))
    assert [s[0] for s in seen] == [False, True, True, False, True]  # cold, warm, warm, guard trips, warm
    assert seen[1][1] < seen[0][1] and seen[2][1] < seen[0][1]


# ---------------------------------------------------------------- thread-block solver
def _solve_block(lib, r2o, w, fixed, max_iters=24, tol=1e-4, anchor=None, valid=None, guard=0.1):
    g, d = r2o.shape
    nb = w.shape[0]
    r = np.ascontiguousarray(r2o.numpy().astype(np.int32))
    o = np.ascontiguousarray(topology.invert_r2o(r2o).numpy().astype(np.int32))
    wa = np.ascontiguousarray(w.numpy().astype(np.float64))
    fa = np.ascontiguousarray(fixed.numpy().astype(np.float64))
    f = np.zeros((nb, g, d))
    iters = np.zeros(nb, np.int32)
    conv = np.zeros(nb, np.int32)
    ptr = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    rc = lib.lplb_sim_solve_block(g, d, ptr(r), ptr(o), nb, ptr(wa), ptr(fa), max_iters, ctypes.c_double(tol), ptr(f),
                                  ptr(iters), ptr(conv), ptr(anchor), ptr(valid), ctypes.c_double(guard),
                                  ctypes.c_double(1e-3))
    assert rc == 0
    return torch.from_numpy(f), iters, conv


@pytest.mark.parametrize("name,nb", [
    ("cube", 2), ("ring5", 2), ("hypercube", 2), ("torus8x4", 2), ("torus8x8", 1), ("ring41", 1),
    ("circ12x3", 1), ("circ10x5", 1),
])
def test_block_solver_device_code_matches_the_torch_restatement(sim, name, nb):
    """The thread-block solver's device code under the block emulation (256 threads, block
    and named barriers, shared memory as a host buffer): one warp of ranks, several warps of
    ranks, group sizes that are not multiples of 8, and the padded replica count."""
    if name == "circ12x3":
        r2o = topology.circulant(12, (1, 2, 5))
    elif name == "circ10x5":
        r2o = topology.circulant(10, (1, 2, 3, 4, 5))
    else:
        r2o = topology.by_name(name)
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(7)
    cnt = ((torch.randn(nb, g, d + 6, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
    f, iters, conv = _solve_block(sim, r2o, w, fixed)
    ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4)
    assert conv.all() and bool(((f >= 0) & (f <= 1)).all())
    if d <= 4:  # the padded variant carries extra (empty) variables, so its path differs slightly
        assert iters.tolist() == ref.iters.tolist()
        assert float((f - ref.f).abs().max()) < 1e-5
    for i in range(nb):
        _, t_opt = lp.solve_highs(w[i], fixed[i], r2o)
        mine = float(lp.rank_loads(f[i], w[i], fixed[i], r2o).max())
        assert -1e-9 < (mine - t_opt) / t_opt < 1e-3


def test_block_solver_handles_empty_groups_and_the_iteration_cap(sim):
    r2o = topology.hypercube()
    w = torch.zeros(1, 16, 2, dtype=torch.float64)
    fixed = torch.zeros(1, 16, dtype=torch.float64)
    f, iters, conv = _solve_block(sim, r2o, w, fixed)
    assert conv[0] == 1 and iters[0] == 0 and torch.equal(f, torch.ones(1, 16, 2, dtype=torch.float64))
    w = torch.rand(1, 16, 2, dtype=torch.float64, generator=torch.Generator().manual_seed(1)) * 1000
    fixed = torch.rand(1, 16, dtype=torch.float64, generator=torch.Generator().manual_seed(2)) * 1000
    f, iters, conv = _solve_block(sim, r2o, w, fixed, max_iters=1, tol=1e-9)
    assert conv[0] == 0 and iters[0] == 1 and bool(((f >= 0) & (f <= 1)).all())


def test_block_solver_warm_start_follows_the_torch_restatement(sim):
    r2o = topology.torus(8, 4)
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(13)
    mean = (torch.rand(g, 8, generator=gen, dtype=torch.float64) + 0.5) * 4096
    anchor_c = np.zeros((1, g, 4 * d + 3))
    valid_c = np.zeros(1, np.int32)
    anchor_t = None
    seen = []
    for step in range(4):
        if step == 3:
            mean = mean.flip(0) * torch.linspace(0.3, 2.0, 8, dtype=torch.float64)
        cnt = (mean * (1 + 0.02 * torch.randn(g, 8, generator=gen, dtype=torch.float64))).floor().unsqueeze(0)
        w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
        ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4, warm_start=True, anchor=anchor_t, guard=0.1)
        anchor_t = ref.anchor
        f, iters, conv = _solve_block(sim, r2o, w, fixed, anchor=anchor_c, valid=valid_c)
        assert conv[0] == 1 and int(iters[0]) == int(ref.iters[0])
        assert float((f - ref.f).abs().max()) < 1e-5
        seen.append((bool(ref.warm[0]), int(iters[0])))
    assert [s[0] for s in seen] == [False, True, True, False]
    assert seen[1][1] < seen[0][1]


def test_solver_sources_are_clean_under_address_and_undefined_behaviour_sanitizers(tmp_path):
    """The solvers' device code, compiled for the host with -fsanitize=address,undefined and run
    on a few instances in a child process: out-of-bounds shared-memory indices, misaligned
    accesses and signed overflow in the index arithmetic would abort the child."""
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "sim_asan"
    main_cpp = tmp_path / "main.cpp"
    main_cpp.write_text(r'''
#include <cstdio>
#include <vector>
extern "C" int lplb_sim_solve_block(int, int, const int*, const int*, int, const double*, const double*, int, double,
                                    double*, int*, int*, double*, int*, double, double);
extern "C" int lplb_sim_solve(int, int, const int*, const int*, int, const double*, const double*, int, double, double*,
                              int*, int*);
extern "C" int lplb_sim_solve_tiles(int, int, int, const int*, const int*, int, const double*, const double*, int, double,
                                    double*, int*, int*, double*, int*, double, double);
int main() {
  int bad = 0;
  for (int g : {5, 8, 19, 40}) {
    std::vector<int> r2o(g), o2r(g);
    for (int i = 0; i < g; ++i) { r2o[i] = (i + 1) % g; o2r[(i + 1) % g] = i; }
    std::vector<double> w(g), fixed(g), f(g);
    for (int i = 0; i < g; ++i) { w[i] = 100.0 + 37.0 * ((i * 7) % 11); fixed[i] = 500.0 + 13.0 * ((i * 5) % 17); }
    int iters = 0, conv = 0;
    std::vector<double> anchor((size_t)g * 7, 0.0);
    int valid = 0;
    for (int rep = 0; rep < 2; ++rep) {
      bad += lplb_sim_solve_block(g, 1, r2o.data(), o2r.data(), 1, w.data(), fixed.data(), 24, 1e-4, f.data(), &iters,
                                  &conv, anchor.data(), &valid, 0.1, 1e-3);
      bad += conv != 1;
    }
    // the tile solver, with one replica and with three (four lanes a rank, one of them a dummy)
    valid = 0;
    for (int rep = 0; rep < 2; ++rep) {
      bad += lplb_sim_solve_tiles(g, 1, g, r2o.data(), o2r.data(), 1, w.data(), fixed.data(), 24, 1e-4, f.data(), &iters,
                                  &conv, anchor.data(), &valid, 0.1, 1e-3);
      bad += conv != 1;
    }
    std::vector<int> r2o3(3 * g), o2r3(3 * g);
    std::vector<double> w3(3 * g), f3(3 * g), anchor3((size_t)g * 15, 0.0);
    for (int i = 0; i < g; ++i)
      for (int d = 0; d < 3; ++d) {
        r2o3[3 * i + d] = (i + d + 1) % g;
        o2r3[3 * ((i + d + 1) % g) + d] = i;
        w3[3 * i + d] = w[i] / (d + 1);
      }
    int valid3 = 0;
    for (int rep = 0; rep < 2; ++rep) {
      bad += lplb_sim_solve_tiles(g, 3, g, r2o3.data(), o2r3.data(), 1, w3.data(), fixed.data(), 24, 1e-4, f3.data(), &iters,
                                  &conv, anchor3.data(), &valid3, 0.1, 1e-3);
      bad += conv != 1;
    }
    if (g <= 32) {
      bad += lplb_sim_solve(g, 1, r2o.data(), o2r.data(), 1, w.data(), fixed.data(), 24, 1e-4, f.data(), &iters, &conv);
      bad += conv != 1;
    }
  }
  std::printf("SANITIZED_OK %d\n", bad);
  return bad;
}
''')
    build = subprocess.run(
        ["g++", "-O1", "-g", "-std=c++17", "-pthread", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
         "-fno-omit-frame-pointer", str(CSRC / "sim_solver.cpp"), str(main_cpp), "-o", str(exe)],
        capture_output=True, text=True,
    )
    if build.returncode != 0 and "sanitize" in build.stderr and ("cannot find" in build.stderr or "unrecognized" in build.stderr):
        pytest.skip("host compiler has no sanitizer runtime")
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600,
                         env=dict(__import__("os").environ, ASAN_OPTIONS="detect_leaks=0"))
    assert run.returncode == 0, run.stdout[-1000:] + run.stderr[-3000:]
    assert "SANITIZED_OK 0" in run.stdout


# ---------------------------------------------------------------- tile solver
def _solve_tiles(lib, r2o, w, fixed, rows=None, max_iters=24, tol=1e-4, anchor=None, valid=None, guard=0.1):
    g, d = r2o.shape
    nb = w.shape[0]
    r = np.ascontiguousarray(r2o.numpy().astype(np.int32))
    o = np.ascontiguousarray(topology.invert_r2o(r2o).numpy().astype(np.int32))
    wa = np.ascontiguousarray(w.numpy().astype(np.float64))
    fa = np.ascontiguousarray(fixed.numpy().astype(np.float64))
    f = np.zeros((nb, g, d))
    iters = np.zeros(nb, np.int32)
    conv = np.zeros(nb, np.int32)
    ptr = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    rc = lib.lplb_sim_solve_tiles(g, d, rows or g, ptr(r), ptr(o), nb, ptr(wa), ptr(fa), max_iters, ctypes.c_double(tol),
                                  ptr(f), ptr(iters), ptr(conv), ptr(anchor), ptr(valid), ctypes.c_double(guard),
                                  ctypes.c_double(1e-3))
    assert rc == 0
    return torch.from_numpy(f), iters, conv


@pytest.mark.parametrize("g,offsets", [
    (2, (1,)), (5, (1,)), (8, (1, 4)), (8, (1, 2, 3, 4)), (9, (1, 2)), (16, (3, 8)), (16, (1, 2, 3, 4)), (17, (1,)),
    (32, (1, 16)), (33, (1, 2)), (64, (1, 8)),
    (8, (1, 2, 4)), (12, (1, 5, 7)), (24, (1, 2, 3)), (40, (1, 2, 3)), (64, (1, 2, 3, 4)),
])
def test_tile_solver_device_code_matches_the_torch_restatement(sim, g, offsets):
    """Group sizes at the edges of the tile counts (1, 2, 4 and 8 warps), with rows that are only padding, and
    offsets of half the group, whose two terms fall into one column of the normal matrix.  The
    iterates differ by the rounding of the step lengths (2^-26, times at most seven iterations and
    the conditioning of the last ones); 1e-5 is what the other solvers are held to."""
    r2o = topology.circulant(g, offsets)
    d = r2o.shape[1]
    gen = torch.Generator().manual_seed(7)
    cnt = ((torch.randn(1, g, d + 6, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
    f, iters, conv = _solve_tiles(sim, r2o, w, fixed)
    ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4)
    assert conv.all() and bool(((f >= 0) & (f <= 1)).all())
    assert iters.tolist() == ref.iters.tolist()
    assert float((f - ref.f).abs().max()) < 1e-5
    if g < 8 and d == 1:  # with the padding rows taking part, as in the warp solver
        f8, it8, _ = _solve_tiles(sim, r2o, w, fixed, rows=8)
        ref8, ref_it, _ = _solve(sim, r2o, w, fixed)
        assert it8.tolist() == ref_it.tolist() and float((f8 - ref8).abs().max()) < 1e-5


@pytest.mark.parametrize("name", ["cube", "ring5", "hypercube"])
def test_tile_solver_warm_start_follows_the_torch_restatement(sim, name):
    r2o = topology.by_name(name)
    g, d = r2o.shape
    gen = torch.Generator().manual_seed(13)
    mean = (torch.rand(g, 8, generator=gen, dtype=torch.float64) + 0.5) * 4096
    anchor_c, valid_c, anchor_t = np.zeros((1, g, 4 * d + 3)), np.zeros(1, np.int32), None
    seen = []
    for step in range(4):
        if step == 3:
            mean = mean.flip(0) * torch.linspace(0.3, 2.0, 8, dtype=torch.float64)
        cnt = (mean * (1 + 0.02 * torch.randn(g, 8, generator=gen, dtype=torch.float64))).floor().unsqueeze(0)
        w, fixed = cnt[:, :, :d].contiguous(), cnt[:, :, d:].sum(-1)
        ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4, warm_start=True, anchor=anchor_t, guard=0.1)
        anchor_t = ref.anchor
        f, iters, conv = _solve_tiles(sim, r2o, w, fixed, anchor=anchor_c, valid=valid_c)
        assert conv[0] == 1 and int(iters[0]) == int(ref.iters[0])
        assert float((f - ref.f).abs().max()) < 1e-5
        seen.append((bool(ref.warm[0]), int(iters[0])))
    assert [s[0] for s in seen] == [False, True, True, name == "ring5"]  # the small shift of five loads stays in the guard
    assert seen[1][1] < seen[0][1]


@pytest.mark.parametrize("g,offsets", [(8, (1, 2, 4)), (12, (1, 5, 7)), (24, (1, 2, 3)), (40, (1, 2, 3))])
def test_tile_solver_warm_starts_with_three_replicas(sim, g, offsets):
    """Four lanes share three edges and the saved iterate has no fourth."""
    r2o = topology.circulant(g, offsets)
    gen = torch.Generator().manual_seed(17)
    mean = (torch.rand(g, 8, generator=gen, dtype=torch.float64) + 0.5) * 4096
    anchor_c, valid_c, anchor_t = np.zeros((1, g, 15)), np.zeros(1, np.int32), None
    for step in range(2):
        cnt = (mean * (1 + 0.02 * torch.randn(g, 8, generator=gen, dtype=torch.float64))).floor().unsqueeze(0)
        w, fixed = cnt[:, :, :3].contiguous(), cnt[:, :, 3:].sum(-1)
        ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4, warm_start=True, anchor=anchor_t, guard=0.1)
        anchor_t = ref.anchor
        f, iters, conv = _solve_tiles(sim, r2o, w, fixed, anchor=anchor_c, valid=valid_c)
        assert conv[0] == 1 and int(iters[0]) == int(ref.iters[0]) and bool(ref.warm[0]) == (step == 1)
        assert float((f - ref.f).abs().max()) < 1e-5


def test_tile_solver_warm_start_with_nearly_singular_systems(sim):
    """Two batches of a skewed gate: one loaded expert per rank, second bundles empty, so that the four most
    loaded ranks are a part of their own whose normal matrix is singular up to s / y.  The second
    solve starts from the iterate of the first and takes as long as the restatement does."""
    r2o = topology.cube()
    heavy = torch.tensor([[675, 452, 385, 314, 313, 307, 275, 211], [640, 471, 374, 332, 306, 280, 279, 221]], dtype=torch.float64)
    rest = torch.tensor([[0, 0, 0, 0, 0, 0, 0, 2], [0, 0, 0, 0, 0, 0, 1, 1]], dtype=torch.float64)
    anchor_c, valid_c, anchor_t = np.zeros((1, 8, 11)), np.zeros(1, np.int32), None
    for step in range(2):
        w, fixed = torch.stack([heavy[step], torch.zeros(8, dtype=torch.float64)], -1).unsqueeze(0), rest[step].unsqueeze(0)
        ref = lp.solve_ipm(w, fixed, r2o, tol=1e-4, warm_start=True, anchor=anchor_t, guard=0.1)
        anchor_t = ref.anchor
        f, iters, conv = _solve_tiles(sim, r2o, w, fixed, rows=8, anchor=anchor_c, valid=valid_c)
        assert conv[0] == 1 and int(iters[0]) == int(ref.iters[0])
        assert float((f - ref.f).abs().max()) < 1e-5


@pytest.mark.parametrize("g,offsets", [(8, (1, 4)), (16, (3, 8)), (64, (1, 8))])
def test_tile_solver_reaches_small_tolerances(sim, g, offsets):
    """A gap of 1e-7, three orders below the default: the systems of the last iterations are the worse conditioned."""
    r2o = topology.circulant(g, offsets)
    gen = torch.Generator().manual_seed(3)
    cnt = ((torch.randn(1, g, 8, generator=gen, dtype=torch.float64) * 0.3 + 1).clamp_min(0) * 4096).floor()
    w, fixed = cnt[:, :, :2].contiguous(), cnt[:, :, 2:].sum(-1)
    f, iters, conv = _solve_tiles(sim, r2o, w, fixed, tol=1e-7)
    ref = lp.solve_ipm(w, fixed, r2o, tol=1e-7)
    assert bool(ref.converged.all()) and conv[0] == 1 and int(iters[0]) <= int(ref.iters[0]) + 1
    best = lp.solve_ipm(w, fixed, r2o, tol=1e-9, max_iters=60)
    realised = float(lp.rank_loads(f, w, fixed, r2o).max())
    assert realised <= float(best.t[0]) * (1 + 2e-7)


def test_tile_solver_handles_empty_groups_and_the_iteration_cap(sim):
    for r2o in (topology.cube(), topology.hypercube()):
        g, d = r2o.shape
        zero = torch.zeros(1, g, d, dtype=torch.float64)
        f, iters, conv = _solve_tiles(sim, r2o, zero, zero[:, :, 0])
        assert conv[0] == 1 and iters[0] == 0 and torch.equal(f, torch.ones(1, g, d, dtype=torch.float64))
        w = torch.rand(1, g, d, dtype=torch.float64, generator=torch.Generator().manual_seed(1)) * 1000
        fixed = torch.rand(1, g, dtype=torch.float64, generator=torch.Generator().manual_seed(2)) * 1000
        f, iters, conv = _solve_tiles(sim, r2o, w, fixed, max_iters=1, tol=1e-9)
        assert conv[0] == 0 and iters[0] == 1 and bool(((f >= 0) & (f <= 1)).all())


def _step_keys(lib, x, limit):
    x = np.ascontiguousarray(x, dtype=np.float64)
    keys, steps = np.zeros(len(x), np.uint32), np.zeros(len(x))
    lib.lplb_sim_step_keys(len(x), ctypes.c_void_p(x.ctypes.data), ctypes.c_double(limit), ctypes.c_void_p(keys.ctypes.data),
                           ctypes.c_void_p(steps.ctypes.data))
    return keys, steps


def test_step_keys_order_like_their_values_over_the_whole_range(sim):
    """From 2^63 on a key is one of the largest 64, whose step is next to nothing, instead of starting
    over at the small ones; a truncated value is at most 2^-26 of itself too small."""
    rng = np.random.default_rng(0)
    x = np.sort(np.concatenate([[0.5, 0.995, 1.0, 2.0**62, np.nextafter(2.0**63, 0)], 2.0 ** rng.uniform(-1, 63, 2000)]))
    small = [-np.inf, -1e300, -1.0, -0.0, 0.0, 5e-324, 1e-9, 0.25, 0.4999999]
    huge = [2.0**63, 9.3e18, 2.0**64, 1e25, 1e300, np.inf]
    for limit in (1.0, 0.995):
        keys, steps = _step_keys(sim, x, limit)
        assert bool((np.diff(keys.astype(np.int64)) >= 0).all())
        assert float(np.abs(steps * np.maximum(x, limit) / limit - 1).max()) < 2.0**-25
        keys, steps = _step_keys(sim, small, limit)
        assert bool((keys < 64).all()) and bool((steps == 1.0).all())
        keys, steps = _step_keys(sim, huge, limit)
        assert bool((keys >= 2**32 - 64).all()) and bool((steps <= 2.0**-62).all())


def test_reciprocals_hold_their_bounds_from_a_seed_of_twenty_bits(sim):
    """The seed's error is at most 2^-18.4 (input and output cut to 20 bits, and one unit of its own): squared
    below 2^-36 for the ratios behind a step length, which keep 26 bits, and cubed below the roundings of
    1/x, four of 2^-53."""
    rng = np.random.default_rng(1)
    x = 2.0 ** rng.uniform(-400, 400, 20000)
    dx = x * rng.uniform(-3, 3, 20000)
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    inverse, ratio = np.zeros_like(x), np.zeros_like(x)
    sim.lplb_sim_reciprocals(len(x), ptr(x), ptr(dx), ptr(inverse), ptr(ratio))
    assert float(np.abs(inverse * x - 1).max()) < 4 * 2.0**-53
    assert float(np.abs(ratio * x / -dx - 1).max()) < 2.0**-36

"""The same sources and flags give the same device code."""

import shutil
import subprocess

import pytest

from lplb_b200 import _native


def test_nothing_in_the_flags_leaves_the_code_to_chance():
    # split compilation gave one of two device codes for moe_launch.cu, 2 to 3 % apart in the grouped GEMMs
    assert not [f for f in _native.NVCC_FLAGS if "split-compile" in f]


def test_every_planner_source_is_built():
    assert sorted(p.name for p in _native._CSRC.glob("planner_*.cu")) == sorted(s for s in _native.SOURCES if s.startswith("planner_"))


def test_two_builds_of_one_source_are_alike(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("no CUDA compiler")
    outs = [tmp_path / f"{i}.fatbin" for i in range(2)]
    jobs = [
        subprocess.Popen(["nvcc", *_native.NVCC_FLAGS, "-fatbin", f"-I{_native._CSRC}", str(_native._CSRC / "moe_launch.cu"), "-o", str(out)])
        for out in outs
    ]
    assert all(job.wait() == 0 for job in jobs)
    # the order of equal entries in its tables is the compiler's own; their size, and the code's, is not
    assert outs[0].stat().st_size == outs[1].stat().st_size

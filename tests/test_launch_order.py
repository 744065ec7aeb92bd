"""Kernels that start while their predecessor still runs touch no memory before they have waited for it
(checked in the source: what a violation does depends on how far the two kernels overlap)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "lplb_b200" / "csrc"
TEXT = "\n".join(re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*")))
# every kernel that launch_after() is given, by name or through the local `kernel`
EARLY = sorted(set(re.findall(r"launch_after\((\w+_kernel)\b", TEXT)) | {"grouped_gemm_kernel", "tile_solve_kernel"})
ACCESS = re.compile(r"\w+\[[^\]]*\]\s*[-+|]?=(?!=)|\batomic\w+\(|\basm\b|\b_*(ld|st|red)_\w+\(|__ldcg?\(|[;{}]\s*\*\s*\w+\s*=(?!=)")


def _before_the_wait(kernel):
    start = re.search(r"__global__[^;{]*?\b%s\([^{;]*\{" % kernel, TEXT, re.S)
    assert start, kernel
    end = TEXT.index("wait_predecessors();", start.end())
    assert "__global__" not in TEXT[start.end() : end], f"{kernel} does not wait"
    return TEXT[start.end() : end]


@pytest.mark.parametrize("kernel", EARLY)
def test_an_early_kernel_waits_before_its_first_access(kernel):
    found = ACCESS.search(_before_the_wait(kernel))
    assert found is None, f"{kernel}: {found.group(0)}"


def test_all_early_kernels_are_looked_at():
    assert set(EARLY) == {"combine_kernel", "dispatch_kernel", "grouped_gemm_kernel", "route_kernel", "schedule_kernel", "tile_solve_kernel"}

"""Kernels that may be launched as programmatic dependents are resident while the kernel in front still writes: the non-coherent load path
(``__ldg``, ``ld.global.nc``), which holds only for memory that nobody writes meanwhile, must not read what a kernel in front may have
written. A rule about the sources, checked on the sources: no run can show that a guarantee is missing."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tilefish_b200", "csrc")
DEPENDENT = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "griddep_wait()" in open(os.path.join(CSRC, f)).read())
HEADERS = sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh"))


def code(name):
    """The file without its // comments."""
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_the_rule_covers_the_dependent_kernels():
    assert DEPENDENT == ["gemm_blockscaled.cu", "quantize.cu", "rmsnorm.cu"]


@pytest.mark.parametrize("name", DEPENDENT + HEADERS)
def test_nothing_a_predecessor_may_write_is_read_non_coherently(name):
    text = code(name)
    assert "ld.global.nc" not in text
    assert set(re.findall(r"__ldg\(([^)]*)\)", text)) <= {"w + v"}  # the norm weights


def test_the_aligned_cluster_barrier_is_reached_by_whole_warps():
    text = code("gemm_blockscaled.cu")
    assert len(re.findall(r"barrier\.cluster\.(?:arrive|wait)", text)) == 2  # both in one place
    assert re.search(r"void cluster_sync_all\(\) \{\s*__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.arrive", text)


def test_a_flag_of_another_warp_is_read_by_vote():
    """Lanes that branch on what each of them reads of a word another warp is storing may leave a loop of warp operations at different turns."""
    reads = re.findall(r"^.*\*started_flag\b(?! = ).*$", code("gemm_blockscaled.cu"), re.M)
    reads = [r.strip() for r in reads if "volatile" not in r]
    assert reads == ["if (__any_sync(0xFFFFFFFFu, *started_flag)) left = 0;"]

"""The K ranges of few-row GEMMs. They are part of a result (an f32 sum in another order moves a last bit, and in a stack of MXFP8 blocks
the next quantization moves with it: two blocks at 2 x 6784 x 22272 differed by 0.017), and they decide which calls the entry points take.
The host-side queries assume 148 SMs without a GPU."""

import os

import pytest

from tilefish_b200 import _native

pytestmark = pytest.mark.skipif(not os.path.exists(_native.LIB_PATH), reason="library not built here")
MXFP8, MXFP4, NVFP4, NONE = 0, 1, 2, 0


@pytest.mark.parametrize("fmt,m,n,k,ranges", [
    (MXFP8, 2, 6784, 22272, 8), (MXFP8, 59, 7552, 16384, 4), (MXFP8, 7, 1544, 15456, 11), (MXFP8, 24, 3200, 24320, 5), (MXFP8, 30, 4736, 8288, 4),
    (MXFP8, 16, 6144, 2560, 3), (MXFP8, 1, 2560, 3072, 6), (NVFP4, 64, 8192, 28672, 4), (MXFP8, 18, 1568, 1408, 1)])
def test_ranges(fmt, m, n, k, ranges):
    assert _native.load().tf_gemm_splits(m, n, k, fmt, NONE) == ranges


def test_shapes_that_leave_partial_sums_or_fit_the_static_scratch():
    lib = _native.load()
    assert lib.tf_gemm_splits(58, 8456, 7456, MXFP4, NONE) > 1  # tf_gemm_blockscaled_partials takes it
    assert lib.tf_gemm_splits(52, 7936, 3584, MXFP8, NONE) > 1  # so does the fused decode step of such a stack
    assert lib.tf_gemm_workspace_bytes(11, 38960, 24032, MXFP8, NONE) <= lib.tf_gemm_static_scratch_bytes()


@pytest.fixture
def margin():
    lib = _native.load()
    yield lambda sms: _native.check(lib.tf_set_sm_margin(sms), "tf_set_sm_margin")
    _native.check(lib.tf_set_sm_margin(0), "tf_set_sm_margin")


@pytest.mark.parametrize("fmt,m,n,k,epi", [("nvfp4", 2048, 14336, 8192, "silu_gate"), ("mxfp8", 8192, 6144, 2560, "none"), ("mxfp4", 4096, 8192, 14336, "residual")])
def test_cta_pairs_are_left_beside_a_margin(margin, fmt, m, n, k, epi):
    """A pair of CTAs needs two neighbouring SMs, which the kernel beside it need not leave whole."""
    from tilefish_b200 import kernels as K

    assert K.gemm_launch_form(m, n, k, fmt, epi)[:3] == ("pair", 256, 1)
    for sms in (1, 16, 64):
        margin(sms)
        assert K.gemm_launch_form(m, n, k, fmt, epi)[:3] == ("tiles", 256, 1)


def test_programmatic_launch_can_be_switched_off_and_stays_off_beside_a_margin(margin):
    """Waiting CTAs of a dependent GEMM would take the SMs that the margin leaves to another kernel."""
    from tilefish_b200 import kernels as K

    dependent = lambda m: K.gemm_launch_form(m, 6144, 2560, "mxfp8")[3]  # noqa: E731
    try:
        assert dependent(16) and not dependent(512)
        margin(16)
        assert not dependent(16)
        K.set_programmatic_launch(True)
        assert dependent(16) and dependent(512)
        margin(0)
        K.set_programmatic_launch(False)
        assert not dependent(16)
    finally:
        K.set_programmatic_launch(None)
    assert dependent(16)

"""residual_add_rmsnorm over more rows than the GPU holds at once: blocks that walk over several rows, and blocks of one, two and four rows with a last
one that is not full; one to eight vectors per thread with a quantized copy; scales stored as words, as bytes (a pointer without 4-byte
alignment) and in the plain layout. The residual and the copy's bytes are compared exactly, the bf16 result with the tolerance that the
row kernels' other tests have."""

import pytest
import torch

from oracle import blockscaled as O

pytestmark = pytest.mark.gpu
FMTS = ["mxfp8", "mxfp4", "nvfp4"]


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    return kernels


def check(K, fmt, m, d, want_bf16, with_amax, offset=0, layout="swizzled"):
    from tilefish_b200 import _native as N

    x, res, w = O.randn((m, d), m, torch.bfloat16), O.randn((m, d), d), (1 + 0.1 * O.randn((d,), 3)).to(torch.bfloat16)
    r_ref, out_ref = O.residual_add_rmsnorm(x, res, w)
    xg, rg, wg = x.cuda(), res.cuda(), w.cuda()
    out = torch.full((m, d), 7.0, dtype=torch.bfloat16, device="cuda") if want_bf16 else None
    gs = torch.tensor([0.002], device="cuda") if fmt == "nvfp4" else None
    amax = torch.zeros(1, device="cuda") if with_amax else None
    lay = N.SCALES_SWIZZLED if layout == "swizzled" else N.SCALES_PLAIN
    n_codes, n_scales = (m * d // K.ELEMS_PER_BYTE[fmt], K.scale_bytes(fmt, m, d, layout)) if fmt else (0, 0)
    codes, scales = (torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda") for n in (n_codes, n_scales))
    ptr = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
    N.check(N.load().tf_residual_add_rmsnorm(ptr(xg), ptr(rg), ptr(wg), ptr(out), m, d, 1e-6, K.FORMATS[fmt] if fmt else -1, ptr(codes) if fmt else None,
                                             scales.data_ptr() + offset if fmt else None, lay, ptr(gs), ptr(amax), torch.cuda.current_stream().cuda_stream),
            "tf_residual_add_rmsnorm")
    assert torch.equal(rg.cpu(), r_ref)
    if not want_bf16:  # the copy is the copy of the result that the same kernel stores
        out = K.residual_add_rmsnorm(xg, res.cuda(), wg)
    got = out.cpu()
    assert float((got.float() - out_ref.float()).abs().max()) <= 2.0**-7 * float(out_ref.float().abs().max())
    assert float((got != out_ref).float().mean()) <= 1e-4
    if amax is not None:
        assert float(amax) == float(got.float().abs().max())
    if fmt:
        ref_codes, ref_scales, _ = O.quantize(got, fmt, gs.cpu() if gs is not None else None)
        ref_scales = O.swizzle_scales(ref_scales) if layout == "swizzled" else ref_scales
        assert torch.equal(codes[:n_codes].cpu(), ref_codes.reshape(-1)) and torch.equal(scales[offset:offset + n_scales].cpu(), ref_scales.reshape(-1))
        assert bool((codes[n_codes:] == 0xA5).all()) and bool((scales[:offset] == 0xA5).all()) and bool((scales[offset + n_scales:] == 0xA5).all())


# The row counts are one more than a limit of a GPU of 148 SMs.
@pytest.mark.parametrize("fmt,m,d,want_bf16,with_amax", [
    (None, 9473, 8, True, True), ("mxfp8", 9473, 96, True, False), ("mxfp4", 4999, 320, True, True), ("nvfp4", 5001, 256, False, False),  # walking
    (None, 14301, 352, True, False), ("mxfp8", 14301, 352, True, True),  # two rows per block
    ("mxfp4", 37891, 352, True, True),  # four rows per block
    ("mxfp4", 7105, 2560, False, False), ("nvfp4", 4737, 4064, False, False),  # the copy alone: two rows
    ("mxfp8", 2665, 2560, True, True), ("nvfp4", 889, 2560, True, False), ("mxfp8", 889, 4064, False, False),  # one row; walking
    ("mxfp8", 1111, 8192, True, False), ("mxfp4", 600, 8192, True, True),  # two vectors per thread
    ("mxfp8", 741, 16384, True, False), ("mxfp4", 741, 16384, True, True), ("nvfp4", 130, 12320, True, False),  # four
    ("mxfp8", 593, 32768, True, False), ("nvfp4", 33, 32768, True, True), ("mxfp4", 130, 16416, False, False)])  # eight
def test_rows_beyond_what_is_resident(K, fmt, m, d, want_bf16, with_amax):
    check(K, fmt, m, d, want_bf16, with_amax)


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("m,d", [(1, 32), (130, 96), (33, 2592), (257, 480), (889, 352), (5, 8224)])
def test_scales_as_bytes(K, fmt, m, d):
    for offset in (1, 2, 3, 4):
        check(K, fmt, m, d, True, False, offset=offset)
    check(K, fmt, m, d, True, True, layout="plain")
    check(K, fmt, m, d, False, False, offset=1, layout="plain")


def test_narrow_rows_and_the_maximum_keep_the_pace(K):
    """Rows of 64 and 128 columns against rows of 2048 with as many elements (blocks of two rows were bound by their starts: 4.4 and 2.2 times the
    time, walking 2.4 and 1.4), and the maximum's cost with many short rows (one atomic per two rows: 1.31 and 1.9 times the time)."""
    def time(m, d, with_amax=False):
        x, r, w = torch.zeros((m, d), dtype=torch.bfloat16, device="cuda"), torch.ones((m, d), device="cuda"), torch.ones(d, dtype=torch.bfloat16, device="cuda")
        out, amax = torch.empty_like(x), torch.zeros(1, device="cuda") if with_amax else None
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                K.residual_add_rmsnorm(x, r, w, out=out, amax_out=amax)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    wide = time(32768, 2048)
    assert time(524288, 128) <= 1.8 * wide and time(1048576, 64) <= 3.3 * wide
    assert time(65536, 512, True) <= 1.22 * time(65536, 512) and time(131072, 288, True) <= 1.3 * time(131072, 288)

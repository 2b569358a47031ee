"""The quantizer's steps of eight rows x 256 columns at their edges: ragged rows and columns, rows with a stride, swizzled scales stored as words and
as bytes (a scale pointer without 4-byte alignment), plain scales, and the round trip through the amax launch with two steps per warp. Codes
and scales are defined bit for bit, so everything is compared exactly, and nothing around them may be written."""

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


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("layout", ["swizzled", "plain"])
@pytest.mark.parametrize("m,k,offset", [(1, 32, 0), (2, 64, 1), (31, 288, 2), (33, 96, 4), (64, 256, 3), (97, 4128, 16), (127, 544, 0), (129, 224, 1), (257, 800, 4), (385, 2080, 0),
                                        # rows of fewer than 256 columns: two and four lanes, one to four steps
                                        (300, 32, 4), (65, 32, 3), (1025, 64, 0), (17, 64, 2), (300, 96, 0), (129, 128, 4), (40, 128, 1), (300, 160, 0), (33, 160, 2), (127, 192, 4), (1, 224, 0),
                                        (5000, 224, 0)])
def test_against_the_oracle(K, fmt, layout, m, k, offset):
    wide = O.randn((m, k + 48), m + k, torch.bfloat16)
    wide[:, ::37] *= 100.0
    x = wide[:, 16:16 + k]
    codes, scales, gs = O.quantize(x.contiguous(), fmt)
    scales = O.swizzle_scales(scales) if layout == "swizzled" else scales.reshape(-1)
    n_codes, n_scales = codes.numel(), K.scale_bytes(fmt, m, k, layout)
    codes_buf = torch.full((n_codes + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    scales_buf = torch.full((n_scales + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    out = K.BlockScaledTensor(fmt, (m, k), codes_buf[:n_codes].view(m, -1), scales_buf[offset:offset + n_scales],
                              torch.empty(1, device="cuda") if fmt == "nvfp4" else None, layout)
    q = K.quantize(wide.cuda()[:, 16:16 + k], fmt, layout=layout, out=out)
    assert torch.equal(codes_buf[:n_codes].cpu().view_as(codes), codes)
    assert torch.equal(scales_buf[offset:offset + n_scales].cpu(), scales.reshape(-1))
    assert bool((codes_buf[n_codes:] == 0xA5).all()) and bool((scales_buf[:offset] == 0xA5).all()) and bool((scales_buf[offset + n_scales:] == 0xA5).all())
    if fmt == "nvfp4":
        assert q.global_scale.cpu().view(torch.int32).item() == gs.reshape(1).view(torch.int32).item()


@pytest.mark.parametrize("m,k", [(2400, 4128), (4700, 2080), (9000, 8192), (1, 28672)])
def test_the_scale_from_the_amax_launch(K, m, k):
    """Blocks that take two steps (and the large case, where they start after the amax launch): the bytes of the same tensor with its scale given."""
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), generator=g, device="cuda").bfloat16()
    for scale in (1.0, 3.0e-3):
        x.mul_(scale)
        q = K.quantize(x, "nvfp4")
        gs = (x.abs().max().float().cpu() / torch.tensor(2688.0)).reshape(1).cuda()  # divided on the host: one correctly rounded division
        ref = K.quantize(x, "nvfp4", global_scale=gs)
        assert torch.equal(q.global_scale, gs) and torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)


@pytest.mark.parametrize("gs", [0.0, -0.01, 0.003, 1e-30, 1e-38, 1e30, 3e37])
def test_nvfp4_block_scales_at_the_ends_of_their_range(K, gs):
    """Blocks of zeros, signed zeros, subnormal, huge and mixed values under global scales that underflow, saturate or are negative: the reciprocals come
    from a table over the scale bytes, and a product of zero is a block of zero codes whatever its signs."""
    g = torch.Generator().manual_seed(3)
    x = torch.randn((160, 288), generator=g).bfloat16()
    for i, v in enumerate((0.0, -0.0, 9.2e-41, -1e-38, 3.3e38, -3.3e38, 1e-20, 448.0 * 6)):
        x[i::16, :144] = v
    x[8::16] *= 1e30
    x[9::16] *= 1e-30
    codes, scales, _ = O.quantize(x, "nvfp4", torch.tensor([gs]))
    q = K.quantize(x.cuda(), "nvfp4", global_scale=torch.tensor([gs]).cuda())
    assert torch.equal(q.scales.cpu(), O.swizzle_scales(scales)) and torch.equal(q.codes.cpu(), codes)


@pytest.mark.parametrize("fmt", FMTS)
def test_narrow_rows_take_no_longer_than_wide_ones(K, fmt):
    """The same number of elements in rows of 32 to 192 columns and of 256: a step is bound by its instructions, so lanes without data
    show (the ratio was 1.4 at 192 columns, 6 at 32)."""
    def time(k):
        x = torch.zeros((196608 * 256 // k, k), dtype=torch.bfloat16, device="cuda")
        gs = torch.ones(1, device="cuda") if fmt == "nvfp4" else None
        q = K.quantize(x, fmt, global_scale=gs)
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                K.quantize(x, fmt, global_scale=gs, out=q)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    wide = time(256)
    assert max(time(32), time(64), time(96), time(128)) <= 2.0 * wide and time(192) <= 1.25 * wide

"""nvfp4 quantization that derives its own tensor-wide scale (an amax launch and the quantizer) against torch's maximum and, byte for byte, the two-call
form: the same scale, codes and scale bytes over row splits, odd widths, strided rows and the special values of the maximum."""

import pytest
import torch

from oracle import blockscaled as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    return kernels


def same(K, x, layout="swizzled"):
    q = K.quantize(x, "nvfp4", layout=layout)
    gs = K.nvfp4_global_scale(x)
    ref = K.quantize(x, "nvfp4", layout=layout, global_scale=gs)
    assert torch.equal(q.global_scale.view(torch.int32), gs.view(torch.int32))
    expected = x.abs().max().float().reshape(1) / torch.full((1,), 2688.0, device=x.device)
    assert torch.equal(gs, expected) or bool(gs.isnan() & expected.isnan())
    assert torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)
    return q


@pytest.mark.parametrize("m,k", [(1, 32), (2, 96), (5, 16384), (128, 4096), (300, 2080), (1000, 416), (129, 65536), (5000, 1024), (4096, 8192), (70000, 64)])
def test_dynamic_equals_the_two_call_form(K, m, k):
    x = torch.randn((m, k), generator=torch.Generator().manual_seed(m + k)).to(torch.bfloat16)
    q = same(K, x.cuda())
    if m * k <= 1 << 20:
        codes, scales, gs = O.quantize(x, "nvfp4")
        assert torch.equal(q.codes.cpu(), codes) and torch.equal(q.scales.cpu(), O.swizzle_scales(scales)) and float(q.global_scale) == float(gs)


# the ring of flat 4096-element chunks serves dense tensors of 1212416 elements and more (two chunks per SM); its last chunk may be short
@pytest.mark.parametrize("m,k", [(70000, 64), (1217, 1056), (300, 4128), (75776, 16), (75777, 16)])
def test_the_only_maximum_anywhere(K, m, k):
    total = m * k
    x = torch.rand((m, k), generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()
    expected = torch.full((1,), 37.0, device="cuda") / torch.full((1,), 2688.0, device="cuda")
    short = total // 4096 * 4096
    for at in {0, 15, 16, 4095, 4096, total // 2, short - 1, min(short, total - 1), total - 17, total - 16, total - 1}:
        was = x.view(-1)[at].clone()
        x.view(-1)[at] = -37.0
        assert torch.equal(K.nvfp4_global_scale(x), expected), at
        if k % 32 == 0:
            assert torch.equal(K.quantize(x, "nvfp4").global_scale, expected), at
        x.view(-1)[at] = was


@pytest.mark.parametrize("m,k,ld", [(1, 32, 64), (3, 48, 64), (300, 256, 512), (1217, 1056, 1072), (9000, 2080, 4160), (24, 28672, 30000 // 16 * 16), (5, 65536, 131072)])
def test_the_only_maximum_of_strided_rows(K, m, k, ld):
    """Column slices: the maximum in any row and at both ends of a row counts, what lies between the rows does not."""
    wide = torch.full((m, ld), 99.0, dtype=torch.bfloat16, device="cuda")
    x = wide[:, :k]
    x.copy_(torch.rand((m, k), generator=torch.Generator().manual_seed(k)).to(torch.bfloat16))
    expected = torch.full((1,), 37.0, device="cuda") / torch.full((1,), 2688.0, device="cuda")
    for r, c in {(0, 0), (0, k - 1), (m - 1, 0), (m - 1, k - 1), (m // 2, k // 2), (m - 1, k - 16), (m // 3, min(k - 1, 1024))}:
        was = x[r, c].clone()
        x[r, c] = 37.0
        assert torch.equal(K.nvfp4_global_scale(x), expected), (r, c)
        if k % 32 == 0:
            same(K, x)
        x[r, c] = was


@pytest.mark.parametrize("value", [0.0, float("inf"), float("nan"), 3.3895e38, 1e-40])
def test_special_maxima_and_strided_rows(K, value):
    x = torch.randn((300, 512), device="cuda").to(torch.bfloat16)
    if value == 0.0:
        x.zero_()
    x[299, 511] = value
    same(K, x)
    same(K, x[:, :256], layout="plain")


def test_dynamic_in_a_graph_and_on_a_side_stream(K):
    x = torch.randn((512, 4096), device="cuda").to(torch.bfloat16)
    ref = same(K, x)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        a = K.quantize(x, "nvfp4")
    torch.cuda.current_stream().wait_stream(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b = K.quantize(x, "nvfp4")
    x.mul_(2.0)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a.codes, ref.codes) and torch.equal(b.codes, ref.codes) and torch.equal(b.scales, ref.scales)
    assert float(b.global_scale) == 2.0 * float(ref.global_scale)

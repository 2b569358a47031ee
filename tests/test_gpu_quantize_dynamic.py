"""nvfp4 quantization that derives its own tensor-wide scale (an amax launch and the quantizer) against the two-call form, byte for byte: the same
scale, codes and scale bytes over row splits, odd widths, strided rows and the special values of the maximum."""

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
    assert torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)
    return q


@pytest.mark.parametrize("m,k", [(1, 32), (2, 96), (5, 16384), (128, 4096), (300, 2080), (1000, 416), (129, 65536), (5000, 1024), (4096, 8192), (70000, 64)])
def test_dynamic_equals_the_two_call_form(K, m, k):
    x = torch.randn((m, k), generator=torch.Generator().manual_seed(m + k)).to(torch.bfloat16)
    q = same(K, x.cuda())
    if m * k <= 1 << 20:
        codes, scales, gs = O.quantize(x, "nvfp4")
        assert torch.equal(q.codes.cpu(), codes) and torch.equal(q.scales.cpu(), O.swizzle_scales(scales)) and float(q.global_scale) == float(gs)


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

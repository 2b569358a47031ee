"""The padding of swizzled scales is zeroed by the kernel that writes the scales: whatever the buffer held before, the bytes are the
oracle's, padding included. Sizes at the edges of the 128 x 4 tiles; destinations filled with 0xA5 first."""

import pytest
import torch

from oracle import blockscaled as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    return kernels


def dirty(K, fmt, m, k):
    return K.BlockScaledTensor(fmt, (m, k), torch.empty((m, k // K.ELEMS_PER_BYTE[fmt]), dtype=torch.uint8, device="cuda"),
                               torch.full((K.scale_bytes(fmt, m, k),), 0xA5, dtype=torch.uint8, device="cuda"),
                               torch.zeros(1, device="cuda") if fmt == "nvfp4" else None)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,k", [(1, 32), (1, 2560), (127, 160), (128, 96), (129, 128), (300, 2080), (128, 128)])
def test_quantize_zeroes_the_padding(K, fmt, m, k):
    x = O.randn((m, k), m + k, torch.bfloat16)
    q = K.quantize(x.cuda(), fmt, out=dirty(K, fmt, m, k))
    codes, scales, _ = O.quantize(x, fmt)
    assert torch.equal(q.codes.cpu(), codes) and torch.equal(q.scales.cpu(), O.swizzle_scales(scales))


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("m,d", [(1, 2560), (130, 1056), (128, 512)])
def test_rmsnorm_zeroes_the_padding(K, fmt, m, d):
    x, r, w = O.randn((m, d), 1, torch.bfloat16), O.randn((m, d), 2), O.randn((d,), 3, torch.bfloat16)
    out, q = K.residual_add_rmsnorm(x.cuda(), r.cuda(), w.cuda(), quantize_to=fmt, q_out=dirty(K, fmt, m, d))
    ref = K.quantize(out, fmt)
    assert torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("m,n,k", [(1, 288, 256), (130, 416, 288), (300, 1056, 512), (16, 1056, 4096), (1100, 3104, 256)])
def test_gemm_zeroes_the_padding(K, fmt, m, n, k):
    qa = K.quantize(O.randn((m, k), 4, torch.bfloat16).cuda(), fmt)
    qb = K.quantize(O.randn((n, k), 5, torch.bfloat16, scale=k**-0.5).cuda(), fmt)
    out, q = K.gemm_blockscaled(qa, qb, q_out=dirty(K, fmt, m, n))
    ref = K.quantize(out, fmt)
    assert torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)

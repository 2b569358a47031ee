"""``gemm`` of a bf16 activation is one native call over one scratch tensor: the bytes of ``quantize`` followed by ``gemm_blockscaled``, for every
source of the nvfp4 scale, strided rows, a split-K workspace behind the quantized activation, and the refusals of the two calls."""

import pytest
import torch

from oracle import blockscaled as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    return kernels


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,n,k,epi", [(1, 2560, 3072, "none"), (16, 6144, 2560, "none"), (5, 288, 28672, "residual"), (130, 392, 160, "none"), (33, 256, 96, "silu_gate"),
                                       (1000, 3000, 2720, "residual")])
def test_equals_the_two_calls(K, fmt, m, n, k, epi):
    wide = O.randn((m, k + 32), m, torch.bfloat16).cuda()
    b = K.quantize(O.randn((2 * n if epi == "silu_gate" else n, k), n, torch.bfloat16, scale=k**-0.5).cuda(), fmt)
    amax = wide[:, 16:16 + k].abs().max().float().reshape(1)
    sources = [{}, {"a_amax": amax}, {"a_global_scale": amax.cpu().cuda() / 1500}] if fmt == "nvfp4" else [{}]
    for source in sources:
        for a in (wide[:, 16:16 + k], wide[:, 16:16 + k].contiguous()):
            r1, r2 = (O.randn((m, n), 3).cuda() for _ in range(2))
            res = lambda r: r if epi == "residual" else None  # noqa: E731
            q = K.quantize(a, fmt, amax=source.get("a_amax"), global_scale=source.get("a_global_scale"))
            ref = K.gemm_blockscaled(q, b, epilogue=epi, residual=res(r1))
            out = torch.full((m, n + 8), -7.0, dtype=torch.bfloat16, device="cuda")
            top = torch.zeros(1, device="cuda")
            got = K.gemm(a, b, epilogue=epi, residual=res(r2), out=out[:, :n], amax_out=top, **source)
            assert torch.equal(got, ref) and torch.equal(r1, r2) and bool((out[:, n:] == -7.0).all()) and float(top) == float(ref.float().abs().max())
            assert torch.equal(K.gemm(a, b, epilogue=epi, residual=res(r2), **source), ref)


def test_refusals_come_before_anything_is_enqueued(K):
    from tilefish_b200.errors import TilefishPreconditionError as Refused

    a = torch.zeros((4, 64), dtype=torch.bfloat16, device="cuda")
    b = K.quantize(torch.zeros((64, 64), dtype=torch.bfloat16, device="cuda"), "mxfp8")
    plain = K.quantize(torch.zeros((64, 64), dtype=torch.bfloat16, device="cuda"), "mxfp8", layout="plain")
    other = K.quantize(torch.zeros((64, 96), dtype=torch.bfloat16, device="cuda"), "mxfp8")
    ragged = K.quantize(torch.zeros((60, 64), dtype=torch.bfloat16, device="cuda"), "mxfp8")
    for bad in (lambda: K.gemm(a.float(), b), lambda: K.gemm(a.cpu(), b), lambda: K.gemm(a, plain), lambda: K.gemm(a, other), lambda: K.gemm(a, ragged), lambda: K.gemm(a[:, 1:33], b),
                lambda: K.gemm(a, b, epilogue="residual"), lambda: K.gemm(a, b, epilogue="silu_gate"), lambda: K.gemm(a, b, epilogue="tanh"), lambda: K.gemm(None, b),
                lambda: K.gemm(a, b, out=torch.empty((4, 60), dtype=torch.bfloat16, device="cuda"))):
        with pytest.raises(Refused):
            bad()
    assert K.gemm(a[:0], b).shape == (0, 64)

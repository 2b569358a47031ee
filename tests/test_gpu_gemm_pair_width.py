"""Both tile widths of the CTA pair at their edges: 192-column tiles that start in the middle of a 128-row scale tile or at its edge, last tiles of 8 and
of 184 columns (the second scale tile past the end of B), more than one tile per pair, and 256-column tiles in several waves. Bound against
the oracle: one f32 sum rounded to bf16 on both sides in another order, 2**-8 of the largest result; residual, amax and the
quantized copy follow from the bf16 result exactly."""

import pytest
import torch

from oracle import blockscaled as O

pytestmark = pytest.mark.gpu
TOL = 2.0**-8 * 1.01


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    return kernels


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,n,k,width", [(3000, 2120, 672, 192), (3000, 2104, 544, 192), (4999, 1152, 1056, 192), (1000, 3000, 2720, 192), (2600, 2504, 544, 256), (2600, 2528, 1056, 256)])
def test_against_the_oracle(K, fmt, m, n, k, width):
    for epi in ("none", "residual"):
        assert K.gemm_launch_form(m, n, k, fmt, epi)[:2] == ("pair", width)
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((n, k), n, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    oa, ob = O.quantize(a, fmt), O.quantize(w, fmt)
    ref = O.dequantize(oa[0], oa[1], fmt, oa[2]) @ O.dequantize(ob[0], ob[1], fmt, ob[2]).t()
    res, amax = O.randn((m, n), 7), torch.zeros(1, device="cuda")
    wide = torch.full((m, n + 16), -7.0, dtype=torch.bfloat16, device="cuda")
    out = K.gemm_blockscaled(qa, qb, out=wide[:, :n], amax_out=amax)
    assert float((out.cpu().float() - ref).abs().max()) <= TOL * float(ref.abs().max())
    assert bool((wide[:, n:] == -7.0).all()) and float(amax) == float(out.float().abs().max())
    r, amax = res.cuda(), torch.zeros(1, device="cuda")
    again = K.gemm_blockscaled(qa, qb, epilogue="residual", residual=r, amax_out=amax)
    assert torch.equal(again, out) and torch.equal(r.cpu(), res + out.cpu().float()) and float(amax) == float(out.float().abs().max())
    if fmt != "nvfp4" and n % 32 == 0:
        for want in (True, False):
            o, q = K.gemm_blockscaled(qa, qb, quantize_out=True, want_bf16=want)
            ref_q = K.quantize(out, fmt)
            assert (o is None or torch.equal(o, out)) and torch.equal(q.codes, ref_q.codes) and torch.equal(q.scales, ref_q.scales)

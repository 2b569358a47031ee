"""The forms one GEMM call can be launched in (128-column tiles, K ranges over a cluster of CTAs, the CTA pair) at the edges of their tiles.

Bound against the oracle: both sides round one f32 sum to bf16 and differ by the order of the sum, 2**-8 of the largest result (the
GEMM tests' own bound). Residual, amax and the quantized copy follow from the bf16 result exactly."""

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


SHAPES = [(1, 2560, 3072), (33, 264, 4096), (128, 136, 2080), (129, 1000, 1024), (300, 1024, 4128), (257, 392, 8192), (700, 520, 2048), (1024, 1024, 512),
          (200, 2048, 1024), (513, 4104, 288), (1100, 3104, 544), (100, 20512, 288), (300, 12512, 160)]


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_every_form_meets_the_oracle(K, fmt, m, n, k):
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((n, k), n, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    amax, res = torch.zeros(1, device="cuda"), O.randn((m, n), 7)
    wide = torch.full((m, n + 16), -7.0, dtype=torch.bfloat16, device="cuda")
    out = K.gemm_blockscaled(qa, qb, out=wide[:, :n], amax_out=amax)
    oa, ob = O.quantize(a, fmt), O.quantize(w, fmt)
    ref = O.dequantize(oa[0], oa[1], fmt, oa[2]) @ O.dequantize(ob[0], ob[1], fmt, ob[2]).t()
    assert float((out.cpu().float() - ref).abs().max()) <= TOL * float(ref.abs().max())
    assert bool((wide[:, n:] == -7.0).all()) and float(amax) == float(out.float().abs().max())
    r = res.cuda()
    again = K.gemm_blockscaled(qa, qb, epilogue="residual", residual=r)
    assert float((again.cpu().float() - ref).abs().max()) <= TOL * float(ref.abs().max())
    if K.gemm_launch_form(m, n, k, fmt)[2] == K.gemm_launch_form(m, n, k, fmt, "residual")[2]:  # the same K ranges, the same sums
        assert torch.equal(again, out)
    assert torch.equal(again, K.gemm_blockscaled(qa, qb, epilogue="residual", residual=res.cuda())), "deterministic"
    assert torch.equal(r.cpu(), res + again.cpu().float())
    if fmt != "nvfp4" and n % 32 == 0:
        o, q = K.gemm_blockscaled(qa, qb, quantize_out=True)
        ref_q = K.quantize(o, fmt)
        assert torch.equal(q.codes, ref_q.codes) and torch.equal(q.scales, ref_q.scales)


def test_the_shapes_above_take_every_form(K):
    forms = {fmt: [K.gemm_launch_form(m, n, k, fmt, epi)[:2] for m, n, k in SHAPES for epi in ("none", "residual")] for fmt in ("mxfp8", "mxfp4", "nvfp4")}
    for got in forms.values():
        assert {("tiles", 128), ("tiles", 256), ("cluster", 128), ("pair", 256)} <= set(got)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,n,k", [(2600, 3592, 544), (2600, 3624, 288)])
def test_pairs_that_take_more_than_one_tile(K, fmt, m, n, k):
    """165 tiles on 74 pairs: the second accumulator, its held columns and the staging boxes' reuse, with every epilogue, against the oracle."""
    assert K.gemm_launch_form(m, n, k, fmt)[0] == K.gemm_launch_form(m, n, k, fmt, "residual")[0] == "pair"
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((n, k), n, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    oa, ob = O.quantize(a, fmt), O.quantize(w, fmt)
    ref = O.dequantize(oa[0], oa[1], fmt, oa[2]) @ O.dequantize(ob[0], ob[1], fmt, ob[2]).t()
    res, amax = O.randn((m, n), 7), torch.zeros(1, device="cuda")
    r = res.cuda()
    wide = torch.full((m, n + 16), -7.0, dtype=torch.bfloat16, device="cuda")
    out = K.gemm_blockscaled(qa, qb, epilogue="residual", residual=r, out=wide[:, :n], amax_out=amax)
    assert float((out.cpu().float() - ref).abs().max()) <= TOL * float(ref.abs().max())
    assert bool((wide[:, n:] == -7.0).all()) and float(amax) == float(out.float().abs().max())
    assert torch.equal(r.cpu(), res + out.cpu().float())
    assert torch.equal(K.gemm_blockscaled(qa, qb), out)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("m,n,k,tiles", [(16, 38400, 544, 300), (100, 38392, 1056, 300), (40000, 128, 288, 313), (39937, 120, 544, 313), (40000, 32, 544, 313),
                                         (40000, 24, 544, 313), (39937, 8, 1056, 313)])  # up to 24 columns: from the accumulator, no boxes
def test_residual_tiles_of_128_columns_more_than_one_per_cta(K, fmt, m, n, k, tiles):
    """300 and 313 tiles on 148 CTAs: the staging boxes are filled again while the next tile's sums are formed, in one ring stage fewer."""
    form = K.gemm_launch_form(m, n, k, fmt, "residual")
    assert form[:3] == ("tiles", 128, 1) and -(-m // 128) * -(-n // 128) == tiles
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((n, k), n, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    oa, ob = O.quantize(a, fmt), O.quantize(w, fmt)
    ref = O.dequantize(oa[0], oa[1], fmt, oa[2]) @ O.dequantize(ob[0], ob[1], fmt, ob[2]).t()
    res, amax = O.randn((m, n), 7), torch.zeros(1, device="cuda")
    r = res.cuda()
    wide = torch.full((m, n + 16), -7.0, dtype=torch.bfloat16, device="cuda")
    out = K.gemm_blockscaled(qa, qb, epilogue="residual", residual=r, out=wide[:, :n], amax_out=amax)
    assert float((out.cpu().float() - ref).abs().max()) <= TOL * float(ref.abs().max())
    assert bool((wide[:, n:] == -7.0).all()) and float(amax) == float(out.float().abs().max())
    assert torch.equal(r.cpu(), res + out.cpu().float())


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("k_bytes", [544, 1920, 2048, 2080])  # 5, 15, 16 and 17 stages: from 16 on the load warps take them in turn
def test_gated_pairs_that_take_more_than_one_tile(K, fmt, k_bytes):
    m, f, k = 2600, 1920, k_bytes if fmt == "mxfp8" else 2 * k_bytes
    assert K.gemm_launch_form(m, f, k, fmt, "silu_gate")[0] == "pair"
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((2 * f, k), f, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    oa, ob = O.quantize(a, fmt), O.quantize(w, fmt)
    t = O.f32_to_bf16(O.dequantize(oa[0], oa[1], fmt, oa[2]) @ O.dequantize(ob[0], ob[1], fmt, ob[2]).t())
    out = K.gemm_blockscaled(qa, qb, epilogue="silu_gate")
    top = float(t.float().abs().max())
    # the bound of the gate test below, and the unfused kernels on the same sums bit for bit
    assert float((out.cpu().float() - O.silu_gate(t[:, :f], t[:, f:]).float()).abs().max()) <= 2 * TOL * top * (top + 1.0)
    assert torch.equal(K.silu_gate(K.gemm_blockscaled(qa, qb)), out)
    if fmt != "nvfp4":
        o, q = K.gemm_blockscaled(qa, qb, epilogue="silu_gate", quantize_out=True)
        ref = K.quantize(o, fmt)
        assert torch.equal(o, out) and torch.equal(q.codes, ref.codes) and torch.equal(q.scales, ref.scales)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("m,n,k", [(40, 1056, 16384), (5, 288, 28672), (64, 8192, 28672)])
def test_the_planes_reduction_quantizes_its_output(K, fmt, m, n, k):
    """Planes and the reduction launch (more ranges than a cluster holds, or more tiles than clusters fit): the quantized copy and the
    padding of its scales, over a buffer that held other bytes."""
    assert K.gemm_launch_form(m, n, k, fmt)[0] == "planes"
    qa = K.quantize(O.randn((m, k), m, torch.bfloat16).cuda(), fmt)
    qb = K.quantize(O.randn((n, k), n, torch.bfloat16, scale=k**-0.5).cuda(), fmt)
    dirty = K.BlockScaledTensor(fmt, (m, n), torch.empty((m, n // K.ELEMS_PER_BYTE[fmt]), dtype=torch.uint8, device="cuda"),
                                torch.full((K.scale_bytes(fmt, m, n),), 0xA5, dtype=torch.uint8, device="cuda"))
    out, q = K.gemm_blockscaled(qa, qb, q_out=dirty)
    codes, scales, _ = O.quantize(out.cpu(), fmt)
    assert torch.equal(out, K.gemm_blockscaled(qa, qb))
    assert torch.equal(q.codes.cpu(), codes) and torch.equal(q.scales.cpu(), O.swizzle_scales(scales))


@pytest.mark.parametrize("fmt", ["mxfp8", "nvfp4"])
@pytest.mark.parametrize("m,f,k", [(300, 128, 8192), (1317, 768, 4096), (257, 256, 2080), (1000, 640, 1024)])
def test_gate_over_a_cluster_and_a_pair(K, fmt, m, f, k):
    a, w = O.randn((m, k), m, torch.bfloat16), O.randn((2 * f, k), f, torch.bfloat16, scale=k**-0.5)
    qa, qb = K.quantize(a.cuda(), fmt), K.quantize(w.cuda(), fmt)
    out = K.gemm_blockscaled(qa, qb, epilogue="silu_gate")
    t = K.gemm_blockscaled(qa, qb).float()
    ref = K.silu_gate(t.to(torch.bfloat16)).float()
    # the gate reads two bf16 results that may differ by one rounding (2**-8 of the largest): |silu'| < 1.1, times the other factor
    bound = 2 * TOL * float(t.abs().max()) * (float(t.abs().max()) + 1.0)
    assert float((out.float() - ref).abs().max()) <= bound


@pytest.fixture
def margin():
    """Sets the SM margin; 0 again afterwards."""
    from tilefish_b200 import _native as N

    def set_margin(sms):
        N.check(N.load().tf_set_sm_margin(sms), "tf_set_sm_margin")

    yield set_margin
    set_margin(0)


@pytest.mark.parametrize("m,n,k,epi", [(520, 1064, 4960, "none"), (520, 1064, 4960, "residual"), (1, 1568, 1408, "none"), (384, 640, 8192, "silu_gate"),
                                       (700, 1024, 16384, "none"), (1024, 2304, 512, "none")])
def test_the_margin_does_not_change_a_byte(K, margin, m, n, k, epi):
    """The SM margin is a matter of occupancy: K is cut into the same ranges, so the sums are the same (MXFP8: the sums round)."""
    qa = K.quantize(O.randn((m, k), m, torch.bfloat16).cuda(), "mxfp8")
    qb = K.quantize(O.randn((2 * n if epi == "silu_gate" else n, k), n, torch.bfloat16, scale=k**-0.5).cuda(), "mxfp8")
    results = []
    for sms in (0, 16, 32, 64):
        margin(sms)
        res = O.randn((m, n), 7).cuda() if epi == "residual" else None
        results.append((K.gemm_launch_form(m, n, k, "mxfp8", epi)[2], K.gemm_blockscaled(qa, qb, epilogue=epi, residual=res), res))
    assert results[0][0] > 1 or k == 512
    for ranges, out, res in results[1:]:
        assert ranges == results[0][0] and torch.equal(out, results[0][1])
        assert res is None or torch.equal(res, results[0][2])

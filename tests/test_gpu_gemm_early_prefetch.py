"""GEMMs of at most 128 rows launched as dependents ask their weights into L2 before the kernel in front has completed. Here that kernel is the
one that writes these weights, or the activation: the result must be that of plain launches, byte for byte, at the edges of what is
prefetched (fewer K stages than the limit, ragged K and N, K ranges over planes and clusters, more than one tile per CTA). Every role of the
kernel waits for the kernel in front by itself, so both operands are rewritten in turn."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from tilefish_b200 import kernels

    kernels.require_cuda()
    yield kernels
    kernels.set_programmatic_launch(None)


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "nvfp4"])
@pytest.mark.parametrize("rewritten", ["weights", "activation"])
@pytest.mark.parametrize("m,n,k_bytes,epi,form,tiles", [
    (1, 136, 32, "none", "tiles", 2), (128, 264, 1056, "residual", "tiles", 3), (16, 6144, 2560, "none", "planes", 144), (33, 2568, 8224, "residual", "planes", 147),
    (1, 2560, 3072, "none", "cluster", 120), (64, 20480, 2080, "silu_gate", "tiles", 160), (16, 38400, 544, "residual", "tiles", 300)])
def test_an_operand_written_by_the_kernel_in_front(K, fmt, rewritten, m, n, k_bytes, epi, form, tiles):
    k = k_bytes if fmt == "mxfp8" else 2 * k_bytes  # the same K stages in every format
    g = torch.Generator(device="cuda").manual_seed(n + k)
    rows = 2 * n if epi == "silu_gate" else n
    weights = [torch.randn((rows, k), generator=g, device="cuda").mul_(k**-0.5).bfloat16() for _ in range(2)]
    acts = [torch.randn((m, k), generator=g, device="cuda").bfloat16() for _ in range(2)]
    sources = weights if rewritten == "weights" else acts
    src, qa, qb = torch.empty_like(sources[0]), K.quantize(acts[0], fmt), K.quantize(weights[0], fmt)
    out, res = torch.empty((m, n), dtype=torch.bfloat16, device="cuda"), torch.zeros((m, n), device="cuda")
    ws = torch.empty(max(1, K.gemm_workspace_bytes(m, n, k, fmt, epi)), dtype=torch.uint8, device="cuda")

    def step():
        K.quantize(src, fmt, out=qb if rewritten == "weights" else qa)
        K.gemm_blockscaled(qa, qb, epilogue=epi, residual=res if epi == "residual" else None, out=out, workspace=ws)

    results = {}
    for setting in (False, None):
        K.set_programmatic_launch(setting)
        got = K.gemm_launch_form(m, n, k, fmt, epi)
        assert got[0] == form and got[3] == (setting is None)
        assert -(-rows // got[1]) * got[2] == tiles
        src.copy_(sources[0])
        step()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        seen = []
        for i in range(6):
            src.copy_(sources[i & 1])
            res.zero_()
            graph.replay()
            seen.append((out.clone(), res.clone()))
        results[setting] = seen
    torch.cuda.synchronize()
    for a, b in zip(results[False], results[None]):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    assert not torch.equal(results[None][0][0], results[None][1][0])

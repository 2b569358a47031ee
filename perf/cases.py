"""The work a user of this package has it do, as measurable cases: each goes through the package's public entry points.

Five paths, named by a case's ``path``:

* ``quantize``  ``tilefish_b200.quantize`` of a bf16 [m, k] tensor: weights when a model is loaded, activations before a gemm.
* ``rmsnorm``   ``kernels.residual_add_rmsnorm``, plain or with the quantized copy of its result (``q``).
* ``gemm``      ``kernels.gemm``: bf16 activations (quantized on the fly) against block-scaled weights, with its fused epilogues.
* ``block``     the README decoder block through the typed API: exported plan, replayed eagerly or as one captured CUDA graph.
* ``stack``     ``MlpStack``: several large blocks, called eagerly (prefill) or replayed as one captured CUDA graph (decode).

Inputs are seeded; activations are N(0, 1), weights N(0, 1/sqrt(fan_in)); quantizer inputs have 1 % outliers, as activations do.
"""

import functools
import math
import tempfile

import torch

import tilefish_b200 as tilefish
from tilefish_b200 import Dim, InOut, Tensor, bf16, const, f32
from tilefish_b200 import kernels as K
from tilefish_b200 import mlp as MLP
from tilefish_b200 import runtime

FORMATS = ("mxfp8", "mxfp4", "nvfp4")


def listed():
    return [
        # one MXFP8 linear of a small batch in a loop that is not captured: launches and host work count
        {"name": "gemm_mxfp8_m16", "path": "gemm", "fmt": "mxfp8", "m": 16, "n": 6144, "k": 2560, "epilogue": "none"},
        # a small activation quantized by itself, the tensor-wide NVFP4 scale included
        {"name": "quantize_nvfp4_m128", "path": "quantize", "fmt": "nvfp4", "m": 128, "k": 4096},
        # a prefill's activation in NVFP4: needs the tensor's maximum before the first code
        {"name": "quantize_nvfp4_m8192", "path": "quantize", "fmt": "nvfp4", "m": 8192, "k": 4096},
        # the largest quantization of the sweep (weights of a model being loaded): memory bandwidth
        {"name": "quantize_mxfp8_m65536", "path": "quantize", "fmt": "mxfp8", "m": 65536, "k": 4096},
        # the normalisation alone over a long prefill of a wide model
        {"name": "rmsnorm_m16384_d8192", "path": "rmsnorm", "q": "none", "m": 16384, "d": 8192},
        # ragged sizes in every dimension, added into the residual stream
        {"name": "gemm_mxfp4_ragged_residual", "path": "gemm", "fmt": "mxfp4", "m": 1000, "n": 3000, "k": 2720, "epilogue": "residual"},
        # one NVFP4 linear of a prefill
        {"name": "gemm_nvfp4_m4096", "path": "gemm", "fmt": "nvfp4", "m": 4096, "n": 6144, "k": 2560, "epilogue": "none"},
        # decoding with one sequence through the exported README block: latency
        {"name": "block_mxfp8_m1", "path": "block", "fmt": "mxfp8", "m": 1, "h": 2560, "f": 3072, "captured": True},
        # a medium batch through the same block
        {"name": "block_mxfp8_m512", "path": "block", "fmt": "mxfp8", "m": 512, "h": 2560, "f": 3072, "captured": True},
        # a long prefill through the same block, the plan run without a capture
        {"name": "block_mxfp8_m8192", "path": "block", "fmt": "mxfp8", "m": 8192, "h": 2560, "f": 3072, "captured": False},
        # decoding 64 sequences through 70B-shaped NVFP4 blocks: streaming the weights
        {"name": "stack_nvfp4_decode_m64", "path": "stack", "fmt": "nvfp4", "m": 64, "h": 8192, "f": 28672, "layers": 4, "captured": True},
        # prefill of 4096 tokens through the same blocks: tensor cores
        {"name": "stack_nvfp4_prefill_m4096", "path": "stack", "fmt": "nvfp4", "m": 4096, "h": 8192, "f": 28672, "layers": 2, "captured": False},
    ]


def _spread(rng, lo, hi, step):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    path = rng.choice(("quantize", "rmsnorm", "gemm", "gemm", "block", "stack"))
    fmt = rng.choice(FORMATS)
    if path == "quantize":
        return {"path": path, "fmt": fmt, "m": _spread(rng, 1, 65536, 1), "k": _spread(rng, 256, 8192, 32)}
    if path == "rmsnorm":
        return {"path": path, "q": rng.choice(("none", "mxfp8", "mxfp4")), "m": _spread(rng, 1, 16384, 1), "d": _spread(rng, 512, 8192, 32)}
    if path == "gemm":
        epilogue = rng.choice(("none", "silu_gate", "residual"))
        n = _spread(rng, 256, 16384, 128 if epilogue == "silu_gate" else 8)
        return {"path": path, "fmt": fmt, "m": _spread(rng, 1, 8192, 1), "n": n, "k": _spread(rng, 256, 16384, 32), "epilogue": epilogue}
    m = _spread(rng, 1, 8192 if path == "block" else 4096, 1)
    if path == "block":
        return {"path": path, "fmt": fmt, "m": m, "h": _spread(rng, 1024, 4096, 32), "f": _spread(rng, 1024, 8192, 128), "captured": m <= 512}
    return {"path": path, "fmt": fmt, "m": m, "h": _spread(rng, 2048, 8192, 128), "f": _spread(rng, 4096, 28672, 128), "layers": rng.randint(1, 2), "captured": m <= 256}


# ---- states ----------------------------------------------------------------------------------------------------------------


class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, scale=1.0):
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(generator=self.g)
        return t if scale == 1.0 else t.mul_(scale)

    def outliers(self, *shape):
        t = self.normal(*shape)
        return t.mul_(torch.where(torch.rand(shape, generator=self.g, device="cuda") < 0.01, 100.0, 1.0).to(torch.bfloat16))

    def stream(self, *shape):
        return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(generator=self.g)

    def norm_weight(self, d):
        return (1 + 0.1 * self.stream(d)).to(torch.bfloat16)


@functools.lru_cache(maxsize=None)
def _block_plan(fmt, m, h, f):
    """The README decoder block of one size, and the directory its plan was exported to (kept for the life of the process)."""
    bs = getattr(tilefish, fmt)
    M, H, F = Dim("M", buckets=[m]), Dim("H", h), Dim("F", f)

    @tilefish.kernel
    def residual_add_rmsnorm(x: Tensor[M, H, bf16], residual: InOut[Tensor[M, H, f32]], w: Tensor[H, bf16], *, eps: const[f32] = 1e-6) -> Tensor[M, H, bf16]:
        r = residual + x.to(f32)
        residual[...] = r
        rstd = tilefish.rsqrt(tilefish.mean(r * r, axis=-1, keepdims=True) + eps)
        return (r * rstd * w.to(f32)).to(bf16)

    @tilefish.library("gemm_gu", acc=f32)
    def gemm_gu(a: Tensor[M, H, bf16], b: Tensor[2 * F, H, bs]) -> Tensor[M, 2 * F, bf16]: ...

    @tilefish.library("gemm_d", acc=f32)
    def gemm_d(a: Tensor[M, F, bf16], b: Tensor[H, F, bs]) -> Tensor[M, H, bf16]: ...

    @tilefish.graph(inputs=("x",), weights=("w_n", "w_gu", "w_d"))
    def block(x: Tensor[M, H, bf16], residual: InOut[Tensor[M, H, f32]], w_n: Tensor[H, bf16], w_gu: Tensor[2 * F, H, bs], w_d: Tensor[H, F, bs]):
        n = residual_add_rmsnorm(x, residual, w_n)
        g, u = gemm_gu(n, w_gu).split(F, axis=-1)
        return gemm_d((tilefish.silu(g.to(f32)) * u.to(f32)).to(bf16), w_d)

    directory = tempfile.TemporaryDirectory()
    return block, runtime.export(block, directory.name, overwrite=True), directory


def _weights(r, fmt, h, f):
    """One block's bf16 weights, quantized as a loader does it."""
    return MLP.quantize_weights(r.norm_weight(h), r.normal(2 * f, h, scale=h**-0.5), r.normal(h, f, scale=f**-0.5), fmt)


def prepare(case, seed):
    r = _Random(seed)
    path = case["path"]
    if path == "quantize":
        return {"path": path, "x": r.outliers(case["m"], case["k"]), "fmt": case["fmt"]}
    if path == "rmsnorm":
        m, d = case["m"], case["d"]
        return {"path": path, "x": r.normal(m, d), "residual": r.stream(m, d), "w": r.norm_weight(d), "q": None if case["q"] == "none" else case["q"]}
    if path == "gemm":
        m, n, k, epilogue = case["m"], case["n"], case["k"], case["epilogue"]
        b = r.normal(2 * n if epilogue == "silu_gate" else n, k, scale=k**-0.5)
        residual = r.stream(m, n) if epilogue == "residual" else None
        return {"path": path, "x": r.normal(m, k), "b": K.quantize(b, case["fmt"]), "residual": residual, "epilogue": epilogue}
    m, h, f = case["m"], case["h"], case["f"]
    x, residual = r.normal(m, h), r.stream(m, h)
    if path == "block":
        block, exp, _ = _block_plan(case["fmt"], m, h, f)
        w = _weights(r, case["fmt"], h, f)
        bound = runtime.bind_weights(block, {"w_n": w.w_n, "w_gu": w.w_gu, "w_d": w.w_d}, mode="replay", plan=exp.directory, pin=exp.digest)
        captured = bound.capture(x, residual) if case["captured"] else None
        return {"path": path, "x": x, "residual": residual, "bound": bound, "captured": captured}
    stack = MLP.MlpStack([_weights(r, case["fmt"], h, f) for _ in range(case["layers"])])
    captured = stack.capture(x, residual) if case["captured"] else None
    return {"path": path, "x": x, "residual": residual, "stack": stack, "captured": captured}


def _parts(q):
    return [q.codes, q.scales] + ([q.global_scale] if q.global_scale is not None else [])


def run(state):
    path = state["path"]
    if path == "quantize":
        return _parts(tilefish.quantize(state["x"], state["fmt"]))
    if path == "rmsnorm":
        if state["q"] is None:
            return [K.residual_add_rmsnorm(state["x"], state["residual"], state["w"]), state["residual"]]
        out, q = K.residual_add_rmsnorm(state["x"], state["residual"], state["w"], quantize_to=state["q"])
        return [out, state["residual"], *_parts(q)]
    if path == "gemm":
        y = K.gemm(state["x"], state["b"], epilogue=state["epilogue"], residual=state["residual"])
        return y if state["residual"] is None else [y, state["residual"]]
    if state["captured"] is not None:
        return [state["captured"].replay(), state["residual"]]
    if path == "block":
        return [state["bound"].run(state["x"], state["residual"]), state["residual"]]
    return [state["stack"](state["x"], state["residual"]), state["residual"]]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------


def _quantized_bytes(fmt, rows, k):
    return rows * k * (1 if fmt == "mxfp8" else 0.5) + rows * k / (16 if fmt == "nvfp4" else 32) + (4 if fmt == "nvfp4" else 0)


def work(case):
    path = case["path"]
    if path == "quantize":
        return {"bytes": 2 * case["m"] * case["k"] + _quantized_bytes(case["fmt"], case["m"], case["k"]), "flops": 0}
    if path == "rmsnorm":
        m, d = case["m"], case["d"]
        return {"bytes": 12 * m * d + 2 * d + (0 if case["q"] == "none" else _quantized_bytes(case["q"], m, d)), "flops": 0}
    if path == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        rows = 2 * n if case["epilogue"] == "silu_gate" else n
        out = m * n * (10 if case["epilogue"] == "residual" else 2)
        return {"bytes": 2 * m * k + _quantized_bytes(case["fmt"], rows, k) + out, "flops": 2 * m * rows * k}
    m, h, f, layers = case["m"], case["h"], case["f"], case.get("layers", 1)
    weights = _quantized_bytes(case["fmt"], 2 * f, h) + _quantized_bytes(case["fmt"], h, f) + 2 * h
    return {"bytes": layers * weights + 12 * m * h, "flops": layers * 6 * m * h * f}


def tolerance(case):
    """Measured with the sums in another order: K, H and F permuted by whole scale blocks in both operands, the result put back in order.
    ``max`` is in units of the larger of the value and the rms: one bf16 step is up to 2**-7 of the value."""
    path = case["path"]
    if path == "quantize":
        return "exact"  # codes, scale bytes and the global scale are defined bit for bit
    if path == "rmsnorm":  # seen: rel 3e-5 (single bf16 ties), one step; codes 1.2e-7 (a small tensor's single tie: 8e-6)
        return {"rel": 1.2e-4, "max": 0.03, "differ": 2e-5}
    if path == "gemm":  # seen: rel 3.1e-5, one bf16 step
        return {"rel": 1.2e-4, "max": 0.03}
    if case["fmt"] == "mxfp8":
        # a last bit upstream moves a requantized element by one e4m3 step; seen: one block rel 3.4e-4 at f = 3072, growing with the
        # sums' length (max 0.046); two blocks rel 9.2e-3 at f = 28672, max 0.17
        return {"rel": 4e-3, "max": 0.2} if path == "block" else {"rel": 0.03, "max": 0.6}
    # a last bit upstream moves an e2m1 code, a quarter to a half of the element, and the second block sees it in the whole row;
    # seen over two blocks: rel 4.6e-3, max 0.77
    return {"rel": 0.018, "max": 0.99}

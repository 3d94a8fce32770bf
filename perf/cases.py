"""The performance cases: what a decode step has this package do, through its public entry points.

Weight-only projections for 1 to 16 activation rows in the four stored formats, the 70B-shaped projection stack replayed
from its CUDA graph, the NVFP4 dequantizer, and the activation quantizers. Shapes are those of the package's benchmark
configurations and tests or lie in the ranges these span; values follow the benchmark configurations' distributions.
"""
import math

import torch

import crit_kernels_b200
from crit_kernels_b200 import stack as stacks

DEV = "cuda"
# One 70B-shaped layer: (role, K, N).
ROLES = (("qkv", 8192, 10240), ("o", 8192, 8192), ("gate_up", 8192, 57344), ("down", 28672, 8192))
K_STEP = {"nvfp4": 32, "fp8": 16, "mxfp8": 32, "bf16": 8}          # what each format asks of K
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "fp8": torch.float8_e4m3fn}


def gemv(fmt, m, n, k, x="bf16", out="bf16", blocked=False, **more):
    return {"kind": "gemv", "fmt": fmt, "m": m, "n": n, "k": k, "x": x, "out": out, "blocked": blocked, **more}


def stack(m, layers, swiglu, **more):
    return {"kind": "stack", "m": m, "layers": layers, "swiglu": swiglu, **more}


def listed():
    return [
        # the smallest projection of the benchmark, one token: launch and host time count as much as the bytes
        gemv("nvfp4", 1, 4096, 4096, name="nvfp4_4096_m1"),
        # ragged: K no multiple of a scale tile's width, rows no multiple of anything, cuBLASLt-tiled scales, FP16
        # activations: a checkpoint prepared for a library GEMM, a few sequences at once
        gemv("nvfp4", 5, 2731, 5152, x="fp16", out="fp16", blocked=True, name="nvfp4_tiled_ragged_m5"),
        # FP8 up projection: one token, and eight sequences whose FP32 sums another kernel reads
        gemv("fp8", 1, 28672, 8192, name="fp8_28672x8192_m1"),
        gemv("fp8", 8, 28672, 8192, out="fp32", name="fp8_28672x8192_m8"),
        # MXFP8 at a 13B model's feed-forward shape, speculative decoding of four tokens
        gemv("mxfp8", 4, 13824, 5120, name="mxfp8_13824x5120_m4"),
        # unquantised layers: two sequences, and a full batch of sixteen
        gemv("bf16", 2, 8192, 8192, name="bf16_8192_m2"),
        gemv("bf16", 16, 8192, 8192, name="bf16_8192_m16"),
        # the NVFP4 stack as a decode loop replays it: single stream, and eight rows with SwiGLU between the projections
        stack(1, 4, "", name="stack_m1"),
        stack(8, 3, "fused", name="stack_m8_swiglu"),
        # a stored matrix expanded for a GEMM that takes more rows than the GEMVs do
        {"kind": "dequantize", "n": 8192, "k": 8192, "out": "bf16", "name": "dequantize_8192_bf16"},
        # activations quantised for a W8A8 / W4A4 projection: a decode step's rows, a prompt's rows
        {"kind": "quantize_fp8", "rows": 16, "k": 28672, "name": "quantize_fp8_16x28672"},
        {"kind": "quantize_nvfp4", "rows": 4096, "k": 8192, "name": "quantize_nvfp4_4096x8192"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _rows(rng):
    return min(16, int(_log(rng, 1, 17)))


def draw(rng):
    pick = rng.random()
    if pick < 0.70:      # projections: any format, any row count, widths between an eighth-size shard and gate_up
        fmt = rng.choice(("nvfp4", "nvfp4", "fp8", "mxfp8", "bf16"))
        step = K_STEP[fmt]
        while True:
            # half the widths are what models use (multiples of 256), half are ragged
            n, k = int(_log(rng, 1024, 57344)), int(_log(rng, 1024, 28672))
            if rng.random() < 0.5:
                n, k = max(1024, n // 256 * 256), max(1024, k // 256 * 256)
            k = k // step * step
            if n * k <= 57344 * 8192:
                break
        x = "fp16" if fmt != "bf16" and rng.random() < 0.25 else "bf16"
        return gemv(fmt, _rows(rng), n, k, x=x, out="fp32" if rng.random() < 0.25 else x,
                    blocked=fmt == "nvfp4" and rng.random() < 0.3)
    if pick < 0.82:
        m = _rows(rng)
        return stack(m, rng.randint(1, max(1, min(4, 24 // m))), rng.choice(("", "", "fused", "unfused")))
    if pick < 0.88:
        n, k = int(_log(rng, 1024, 28672)), int(_log(rng, 1024, 28672)) // 16 * 16
        return {"kind": "dequantize", "n": min(n, 28672 * 8192 // k), "k": k, "out": rng.choice(("bf16", "fp16", "fp8"))}
    rows, k = int(_log(rng, 1, 8192)), int(_log(rng, 1024, 28672)) // 16 * 16
    return {"kind": "quantize_fp8" if pick < 0.94 else "quantize_nvfp4", "rows": min(rows, 16384 * 8192 // k), "k": k}


def _fp8_weights(n, k, g):
    return (torch.randn(n, k, device=DEV, generator=g) * 0.02).to(torch.float8_e4m3fn)


def _mxfp8_weights(n, k, g):
    """N(0, 0.02) weights with the MX shared exponent floor(log2(amax)) - 8 per 32."""
    w = torch.randn(n, k // 32, 32, device=DEV, generator=g) * 0.02
    shared = torch.frexp(w.abs().amax(dim=-1))[1] - 9
    codes = (w / torch.exp2(shared.float())[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn)
    return codes.view(n, k), (shared + 127).to(torch.uint8)


def _to_tiles(scales):
    """Row-major [N][blocks] scale bytes in cuBLASLt's 128 x 4 tiles (rows padded to 128, blocks to 4)."""
    n, blocks = scales.shape
    rows, cols = -(-n // 128), -(-blocks // 4)
    padded = torch.zeros(rows * 128, cols * 4, dtype=torch.uint8, device=scales.device)
    padded[:n, :blocks] = scales
    return padded.view(rows, 4, 32, cols, 4).permute(0, 3, 2, 1, 4).contiguous().flatten()


def _prepare_gemv(case, g):
    fmt, m, n, k = case["fmt"], case["m"], case["n"], case["k"]
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    x = torch.randn(m, k, device=DEV, generator=g).to(DTYPES[case["x"]])
    out = torch.empty(m, n, device=DEV, dtype=DTYPES[case["out"]])
    if fmt == "nvfp4":
        codes, scales, inverse = stacks.random_nvfp4(n, k, DEV, g)
        if case["blocked"]:
            scales = _to_tiles(scales)
        return lambda: kernel.gemv(x, codes, scales, inverse, out, blocked=case["blocked"])
    if fmt == "fp8":
        codes = _fp8_weights(n, k, g)
        scales = (torch.rand(n, device=DEV, generator=g) * 1.5 + 0.5) / 64
        return lambda: kernel.gemv_fp8(x, codes, scales, out)
    if fmt == "mxfp8":
        codes, scales = _mxfp8_weights(n, k, g)
        return lambda: kernel.gemv_fp8(x, codes, scales, out)
    w = (torch.randn(n, k, device=DEV, generator=g) * 0.02).to(torch.bfloat16)
    return lambda: kernel.gemv_bf16(x, w, out)


def _prepare_stack(case, g, seed):
    stack_ = stacks.ShardedStack.random(case["layers"], ROLES, 0, 1, torch.device(DEV), seed=seed)
    if case["swiglu"]:
        stack_ = stack_.with_swiglu(case["swiglu"])
        for p in stack_.projections:        # the projections' scales keep the activations near one, as norms do
            p.inverse.fill_(1 / (2 * math.sqrt(p.k)))
    passes = stacks.StackRun(stack_, case["m"])
    for x in passes.x.values():
        x.copy_(torch.randn(x.shape, device=DEV, generator=g).to(x.dtype))
    passes.capture()

    def one_pass():
        passes.replay()
        return passes.outputs()
    return one_pass


def _prepare_dequantize(case, g):
    n, k = case["n"], case["k"]
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    codes, scales, _ = stacks.random_nvfp4(n, k, DEV, g)
    factor = torch.rand(n, device=DEV, generator=g) + 0.5
    out = torch.empty(n, k, device=DEV, dtype=DTYPES[case["out"]])
    call = kernel.decode_fp8 if case["out"] == "fp8" else kernel.decode
    return lambda: call(codes, scales, factor, out)


def _prepare_quantize(case, g):
    rows, k = case["rows"], case["k"]
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    x = torch.randn(rows, k, device=DEV, generator=g).to(torch.bfloat16)
    if case["kind"] == "quantize_fp8":
        q = torch.empty(rows, k, device=DEV, dtype=torch.float8_e4m3fn)
        scale = torch.empty(rows, device=DEV)

        def fp8():
            kernel.quantize_fp8_rows(x, q, scale)
            return q.view(torch.uint8), scale
        return fp8
    codes = torch.empty(rows, k // 2, device=DEV, dtype=torch.uint8)
    tiles = torch.empty(-(-rows // 128) * 128 * (-(-(k // 16) // 4) * 4), device=DEV, dtype=torch.uint8)
    return lambda: kernel.quantize_nvfp4(x, 448 * 6 / 8.0, codes, tiles)


def prepare(case, seed):
    """Inputs made on the GPU from the seed, and the call a program that holds them makes."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    if kind == "gemv":
        return _prepare_gemv(case, g)
    if kind == "stack":
        return _prepare_stack(case, g, seed)
    if kind == "dequantize":
        return _prepare_dequantize(case, g)
    return _prepare_quantize(case, g)


def run(state):
    return state()


def _gemv_work(fmt, m, n, k, x_bytes, out_bytes):
    weights = {"nvfp4": n * k // 2 + n * k // 16 + 4 * n, "fp8": n * k + 4 * n, "mxfp8": n * k + n * k // 32,
               "bf16": 2 * n * k}[fmt]
    return {"bytes": weights + m * k * x_bytes + m * n * out_bytes, "flops": 2 * m * n * k}


def work(case):
    kind = case["kind"]
    if kind == "gemv":
        return _gemv_work(case["fmt"], case["m"], case["n"], case["k"], 2, 4 if case["out"] == "fp32" else 2)
    if kind == "stack":
        total = {"bytes": 0, "flops": 0}
        for role, k, n in ROLES:
            # with SwiGLU, gate_up leaves half its width; without, all of it
            out_bytes = 1 if case["swiglu"] and role == "gate_up" else 2
            for key, v in _gemv_work("nvfp4", case["m"], n, k, 2, out_bytes).items():
                total[key] += case["layers"] * v
        return total
    if kind == "dequantize":
        n, k = case["n"], case["k"]
        return {"bytes": n * k // 2 + n * k // 16 + 4 * n + n * k * (1 if case["out"] == "fp8" else 2), "flops": 2 * n * k}
    rows, k = case["rows"], case["k"]
    out = rows * k + 4 * rows if kind == "quantize_fp8" else rows * k // 2 + rows * k // 16
    return {"bytes": 2 * rows * k + out, "flops": 2 * rows * k}


def tolerance(case):
    """Conversions are exact. Projections: FP32 sums in any order, rounded once to the output type; in the stack with
    SwiGLU a second projection reads the rounded activations of the first."""
    if case["kind"] == "gemv":
        return {"rel": {"fp32": 1e-5, "fp16": 1e-3, "bf16": 5e-3}[case["out"]]}
    if case["kind"] == "stack":
        return {"rel": 1e-2 if case["swiglu"] else 5e-3}
    return "exact"

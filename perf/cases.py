"""The work this library is asked to do, as cases that can be timed and compared: dense products of every stored format
from one activation row to a prefill batch, routed experts for many and for few tokens, and the conversions a loader
runs. Sizes are those of bench.py's workloads and of the tests, and generic ones between them.

A case is a dict of plain values. prepare() makes what a caller holds before the call (stored weights, activations,
workspaces), run() makes one pass through the public entry points (dromos_b200.host, or the C ABI where an option is only
there), work() says what a pass cannot do without, tolerance() how far another correct implementation may be off.
"""

import math

import torch

from dromos_b200 import abi, host

FORMATS = {"bf16": abi.W_BF16, "int8": abi.W_INT8, "fp8": abi.W_FP8, "nvfp4": abi.W_NVFP4, "bf16x": abi.W_BF16X}
# bytes a stored value takes, scales included (BF16X: measured on N(0, 0.02) weights, lx_bf16x_bytes)
VALUE_BYTES = {"bf16": 2.0, "int8": 1.0, "fp8": 1.0, "nvfp4": 0.5625, "bf16x": 1.512}

_lib = None


def library():
    global _lib
    if _lib is None:
        _lib = abi.Library()
    return _lib


def listed():
    return [
        # One row through one small matrix: an attention output projection in a decode step. Latency, launches and the
        # host's share count most.
        {"name": "gemv_bf16", "kind": "dense", "fmt": "bf16", "N": 4096, "K": 4096, "M": 1},
        # A batch of eight sequences through an up projection stored as INT8: the most rows the decode GEMV takes.
        {"name": "gemv_int8_m8", "kind": "dense", "fmt": "int8", "N": 14336, "K": 4096, "M": 8},
        # The lossless format at the same size, one row.
        {"name": "gemv_bf16x", "kind": "dense", "fmt": "bf16x", "N": 14336, "K": 4096, "M": 1},
        # The largest matrix of a decode step, one row, FP8.
        {"name": "gemv_fp8", "kind": "dense", "fmt": "fp8", "N": 28672, "K": 8192, "M": 1},
        # The same matrix for a server's batch of 16 sequences as NVFP4, and of 64 as FP8.
        {"name": "gemm_nvfp4_m16", "kind": "dense", "fmt": "nvfp4", "N": 28672, "K": 8192, "M": 16},
        {"name": "gemm_fp8_m64", "kind": "dense", "fmt": "fp8", "N": 28672, "K": 8192, "M": 64},
        # Ragged everything: rows that divide by nothing, f32 activations, bias, bf16 outputs, accumulation into y.
        {"name": "gemm_ragged", "kind": "product", "fmt": "bf16", "math": 0, "N": 10309, "K": 2304, "M": 37, "x_f32": True, "y_bf16": True,
         "bias": True, "beta": 0.5},
        # Prefill: a prompt of 512 tokens through a bf16 up projection, and one of 1000 with activations quantized to FP8.
        {"name": "prefill_bf16", "kind": "dense", "fmt": "bf16", "N": 14336, "K": 4096, "M": 512},
        {"name": "prefill_fp8_math", "kind": "product", "fmt": "fp8", "math": 2, "N": 14336, "K": 4096, "M": 1000, "x_f32": False,
         "y_bf16": True, "bias": False, "beta": 0.0},
        # Routed experts: 32 decode tokens, routing included (nearly every expert is touched: the largest case), and four
        # tokens through the few-token entry point.
        {"name": "moe_fp8_t32", "kind": "moe", "fmt": "fp8", "E": 64, "top_k": 8, "L": 4096, "I": 1536, "T": 32},
        {"name": "moe_decode_fp8_t4", "kind": "moe_decode", "fmt": "fp8", "E": 64, "top_k": 8, "L": 4096, "I": 1536, "T": 4},
        # What a loader does with one matrix of a checkpoint: encode it losslessly, and decode an encoded one.
        {"name": "convert_bf16x", "kind": "convert", "fmt": "bf16x", "N": 14336, "K": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, fmt, most_n, most_k):
    """Rows and columns of a weight, over their logarithm: any number of rows, columns in the steps the format's layout and
    the entry points ask for (whole scale groups for NVFP4, 16-byte rows for the others)."""
    N = _log_int(rng, 250, most_n)
    step = 256 if fmt == "nvfp4" else 128 if rng.random() < 0.75 else 16
    K = max(512, _log_int(rng, 512, most_k) // step * step)
    return N, K


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "gemv", "gemm", "gemm", "product", "prefill", "prefill", "moe", "moe_decode", "convert"])
    if kind in ("gemv", "gemm", "product", "prefill"):
        fmt = rng.choice(["bf16", "int8", "fp8", "nvfp4", "bf16x"] if kind == "gemv" else ["bf16", "int8", "fp8", "nvfp4"])
        most_n, most_k = (14336, 4096) if kind == "prefill" else (28672, 8192)
        N, K = _matrix(rng, fmt, most_n, most_k)
        if fmt == "bf16x":
            K = K // 128 * 128
        if fmt in ("bf16", "bf16x"):
            N = min(N, 16384)
        M = rng.randint(1, 8) if kind == "gemv" else rng.randint(9, 64) if kind in ("gemm", "product") else _log_int(rng, 65, 1000)
        maths = {"int8": [0, 1], "fp8": [0, 2]}.get(fmt, [0])
        if kind in ("gemv", "gemm"):
            return {"kind": "dense", "fmt": fmt, "N": N, "K": K, "M": M}
        return {"kind": "product", "fmt": fmt, "math": rng.choice(maths), "N": N, "K": K, "M": M, "x_f32": rng.random() < 0.3,
                "y_bf16": rng.random() < 0.5, "bias": rng.random() < 0.5, "beta": rng.choice([0.0, 0.0, 0.5])}
    if kind == "convert":
        fmt = rng.choice(["int8", "fp8", "nvfp4", "bf16x"])
        N, K = _matrix(rng, fmt, 14336, 4096)
        return {"kind": kind, "fmt": fmt, "N": N, "K": K}
    fmt = rng.choice(["bf16", "int8", "fp8", "nvfp4"] if kind == "moe" else ["bf16", "int8", "fp8", "nvfp4", "bf16x"])
    E = rng.choice([8, 16, 32, 64])
    # the stacks of two-byte formats stay within the bytes of the largest FP8 case
    L, I = 256 * _log_int(rng, 1, 16), 256 * _log_int(rng, 1, 3 if fmt in ("bf16", "bf16x") else 6)
    T = _log_int(rng, 9, 64) if kind == "moe" else rng.randint(1, 8)
    return {"kind": kind, "fmt": fmt, "E": E, "top_k": rng.choice([2, 4, 8]), "L": L, "I": I, "T": T}


def _normal(gen, shape, std=1.0):
    out = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    rows = out.view(-1, shape[-1])
    step = max(1, (1 << 26) // shape[-1])  # in pieces: an f32 copy of a whole expert stack would be gigabytes
    for r in range(0, rows.shape[0], step):
        rows[r:r + step] = torch.randn(rows[r:r + step].shape, generator=gen, device="cuda") * std
    return out


def prepare(case, seed):
    lib = library()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = {"lib": lib, "case": case}
    if case["kind"] in ("dense", "product"):
        N, K, M = case["N"], case["K"], case["M"]
        stored = host.store_weight(lib, _normal(gen, (N, K), 0.02), FORMATS[case["fmt"]])
        s["x"] = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
        if case["kind"] == "dense":
            s["layer"] = host.Linear(lib, stored, N, K)
            return s
        s["weight"] = stored
        if case["x_f32"]:
            s["x"] = torch.randn((M, K), generator=gen, device="cuda")
        s["bias"] = torch.randn((N,), generator=gen, device="cuda").to(torch.bfloat16) if case["bias"] else None
        y_dtype = torch.bfloat16 if case["y_bf16"] else torch.float32
        s["residual"] = torch.randn((M, N), generator=gen, device="cuda").to(y_dtype) if case["beta"] else None
        s["y"] = torch.empty((M, N), dtype=y_dtype, device="cuda")
        s["ws"] = torch.empty(lib.lx_gemm_workspace_bytes(M, K, case["math"]), dtype=torch.uint8, device="cuda")
        return s
    if case["kind"] == "convert":
        s["w"] = _normal(gen, (case["N"], case["K"]), 0.02)
        s["back"] = torch.empty_like(s["w"])
        return s
    E, L, I, T, top_k = case["E"], case["L"], case["I"], case["T"], case["top_k"]
    gate_up = host.store_weight(lib, _normal(gen, (E, 2 * I, L), 0.02), FORMATS[case["fmt"]])
    down = host.store_weight(lib, _normal(gen, (E, L, I), 0.02), FORMATS[case["fmt"]])
    s["experts"] = host.Experts(lib, gate_up, down, E, L, I, top_k)
    s["latent"] = torch.randn((T, L), generator=gen, device="cuda").to(torch.bfloat16)
    s["logits"] = torch.randn((T, E), generator=gen, device="cuda")
    if case["kind"] == "moe_decode":
        s["out"] = torch.empty((T, L), dtype=torch.float32, device="cuda")
        s["ws"] = torch.empty(max(256, lib.lx_moe_decode_workspace_bytes(T, I, top_k)), dtype=torch.uint8, device="cuda")
    return s


def _checked(status, what):
    if status:
        raise RuntimeError(f"{what} failed: {status}")


def run(s):
    case, lib = s["case"], s["lib"]
    if case["kind"] == "dense":
        return s["layer"](s["x"])
    if case["kind"] == "product":
        x, y, bias = s["x"], s["y"], s["bias"]
        if s["residual"] is not None:
            y.copy_(s["residual"])
        stream = torch.cuda.current_stream().cuda_stream
        _checked(lib.lx_gemm_w(abi.ptr(x), abi.F32 if case["x_f32"] else abi.BF16, x.stride(0), s["weight"].ref(), case["math"], abi.ptr(bias),
                               abi.BF16, abi.ptr(y), abi.BF16 if case["y_bf16"] else abi.F32, y.stride(0), case["M"], case["N"], case["K"], 1.0,
                               case["beta"], abi.ptr(s["ws"]), stream), "lx_gemm_w")
        return y
    if case["kind"] == "convert":
        w, fmt = s["w"], FORMATS[case["fmt"]]
        stored, stream = host.store_weight(lib, w, fmt), torch.cuda.current_stream().cuda_stream
        if fmt == abi.W_BF16X:
            _checked(lib.lx_bf16x_decode(abi.ptr(stored.data), case["N"], case["K"], abi.ptr(s["back"]), stream), "lx_bf16x_decode")
            return {"data": stored.data, "back": s["back"]}
        _checked(lib.lx_dequantize_weight(stored.ref(), abi.ptr(s["back"]), case["N"], case["K"], stream), "lx_dequantize_weight")
        return {"data": stored.data, "scale": stored.scale, "global": stored.glob, "back": s["back"]}
    experts = s["experts"]
    ids, weights = experts.route(s["logits"])
    if case["kind"] == "moe":
        out = experts(s["latent"], ids, weights)
    else:
        out = s["out"]
        _checked(lib.lx_moe_experts_decode(abi.ptr(s["latent"]), abi.ptr(ids), abi.ptr(weights), experts.gate_up.ref(), experts.down.ref(),
                                           abi.ptr(out), abi.ptr(s["ws"]), case["T"], case["L"], case["I"], case["top_k"],
                                           torch.cuda.current_stream().cuda_stream), "lx_moe_experts_decode")
    return {"ids": ids, "weights": weights, "out": out}


def work(case):
    """Each input read once and each output written once; two operations per weight and row."""
    if case["kind"] in ("dense", "product"):
        N, K, M = case["N"], case["K"], case["M"]
        x = M * K * (4 if case.get("x_f32") else 2)
        y = M * N * (2 if case.get("y_bf16") else 4)
        rows = 4 * N if case["fmt"] in ("int8", "fp8") else 0
        return {"bytes": N * K * VALUE_BYTES[case["fmt"]] + rows + x + (2 * y if case.get("beta") else y) + (2 * N if case.get("bias") else 0), "flops": 2.0 * N * K * M}
    if case["kind"] == "convert":  # the bf16 matrix in, the stored one out and in again, the bf16 matrix out
        return {"bytes": case["N"] * case["K"] * (4 + 2 * VALUE_BYTES[case["fmt"]]), "flops": 0}
    E, L, I, pairs = case["E"], case["L"], case["I"], case["T"] * case["top_k"]
    touched = E * (1 - (1 - case["top_k"] / E) ** case["T"])  # experts some token picks, on average
    return {"bytes": touched * 3 * L * I * VALUE_BYTES[case["fmt"]] + case["T"] * L * 6, "flops": 6.0 * L * I * pairs}


def tolerance(case):
    if case["kind"] == "convert":
        return "exact"  # stored bytes, scales and the values they stand for
    if case["kind"] in ("moe", "moe_decode"):
        # the intermediate row is rounded to bf16 between the two products: another order of the f32 sums moves a few of
        # its values to the neighbouring bf16 number (measured against the same sums in 64 bits: 1.1e-4, largest 2.4e-3)
        return {"rel": 4e-4, "max": 1e-2}
    if case.get("y_bf16"):
        return {"rel": 4e-4, "max": 2e-2}  # f32 sums rounded to bf16: a thousandth land on the neighbouring number, a step of 2^-8 to 2^-7
    # f32 sums; the tensor core's, measured against 64 bits, are off by up to 4.4e-6 (largest 1.6e-5) at K = 4096
    return {"rel": 2e-5, "max": 2e-4}

"""The work a user of this framework has it do, as cases that can be timed and compared.

Kinds of call:

* ``gemm``      ``custom_kernel`` on the 7-tuple with n > 1: the NVFP4 block-scaled matmul;
* ``gemv``      the same entry with n == 1, the memory-bound matrix-vector product;
* ``layer``     a feed-forward block on NVFP4 weights: bf16 or fp16 activations are quantised, go
                through the up projection with bias, SiLU and re-quantisation in its epilogue
                (``gemm_epilogue``), and the down projection (``custom_kernel``) gives fp16;
* ``quantise``  the stand-alone quantiser, fp16 or bf16 to packed e2m1 and both scale layouts.

Operands are what the quantiser makes of normally distributed activations and weights, so that
codes and scales have the distributions that quantised networks have.  Sizes are the benchmark's and
the test suite's own, and generic ones between them.
"""
import torch

from nvfp4_gemm_b200 import _lib
from nvfp4_gemm_b200.inputs import FP4_DTYPE, SF_DTYPE
from nvfp4_gemm_b200.submission import custom_kernel, gemm_epilogue

# What no drawn case goes beyond: the largest listed matmul and the traffic that goes with it.
MOST_FLOPS = 2 * 8192 * 28672 * 8192
MOST_BYTES = 640e6


def listed():
    return [
        # the smallest call of the operator's test shapes: launch and host latency
        {"name": "gemm_smallest", "kind": "gemm", "m": 128, "n": 256, "k": 256, "l": 1},
        # decode with a full 128-row batch of tokens, long K: weights stream through once
        {"name": "gemm_decode_long", "kind": "gemm", "m": 128, "n": 7168, "k": 16384, "l": 1},
        # decode with few tokens in flight: a ragged M far below one tile
        {"name": "gemm_decode_few", "kind": "gemm", "m": 17, "n": 7168, "k": 2048, "l": 1},
        # a chunk of a prompt whose length is no multiple of anything
        {"name": "gemm_chunk_ragged", "kind": "gemm", "m": 1000, "n": 4096, "k": 4096, "l": 1},
        # several independent matmuls in one call, each with a ragged M and a moderate N
        {"name": "gemm_batched", "kind": "gemm", "m": 200, "n": 1536, "k": 2048, "l": 8},
        # prefill, compute bound
        {"name": "gemm_prefill", "kind": "gemm", "m": 4096, "n": 7168, "k": 7168, "l": 1},
        # the largest matmul of the benchmark, on one GPU
        {"name": "gemm_largest", "kind": "gemm", "m": 8192, "n": 28672, "k": 8192, "l": 1},
        # single-token decode: the benchmark's matrix-vector products, long and short rows
        {"name": "gemv_long", "kind": "gemv", "m": 7168, "k": 16384, "l": 4},
        {"name": "gemv_short", "kind": "gemv", "m": 7168, "k": 2048, "l": 4},
        # a feed-forward block while decoding and while reading a prompt
        {"name": "layer_decode", "kind": "layer", "m": 128, "n": 4096, "k": 7168, "bf16": True},
        {"name": "layer_prefill", "kind": "layer", "m": 2048, "n": 4096, "k": 7168, "bf16": True},
        # activations of a long prompt (or weights, once) to NVFP4
        {"name": "quantise_large", "kind": "quantise", "m": 8192, "k": 28672, "bf16": True},
    ]


def _log(rng, low, high):
    return low * (high / low) ** rng.random()


def _multiple(value, step, low):
    return max(low, int(value / step + 0.5) * step)


def draw(rng):
    while True:
        kind = rng.choice(["gemm", "gemm", "gemm", "gemv", "layer", "quantise"])
        if kind == "gemm":
            case = {"kind": kind, "m": int(_log(rng, 1, 8193)), "n": _multiple(_log(rng, 128, 28672), 128, 128),
                    "k": _multiple(_log(rng, 256, 16384), 256, 256), "l": rng.choice([1, 1, 1, 2, 3, 4, 8])}
        elif kind == "gemv":
            case = {"kind": kind, "m": int(_log(rng, 512, 28673)), "k": _multiple(_log(rng, 512, 16384), 64, 512),
                    "l": rng.choice([1, 1, 2, 3, 4, 8])}
        elif kind == "layer":
            case = {"kind": kind, "m": int(_log(rng, 1, 4097)), "n": _multiple(_log(rng, 1024, 16384), 256, 1024),
                    "k": _multiple(_log(rng, 1024, 8192), 256, 1024), "bf16": rng.random() < 0.5}
        else:
            case = {"kind": kind, "m": int(_log(rng, 64, 8193)), "k": _multiple(_log(rng, 512, 28672), 64, 512),
                    "bf16": rng.random() < 0.5}
        need = work(case)
        if need["bytes"] <= MOST_BYTES and need["flops"] <= MOST_FLOPS:
            return case


def _quantise(x, packed, sf, sf_permuted):
    rows, k = x.shape
    _lib.check(_lib.load().nvfp4_quantize(x.data_ptr(), int(x.dtype == torch.bfloat16), packed.data_ptr(), sf.data_ptr(), sf_permuted.data_ptr(),
                                          rows, k, k, k // 2, k // 16, torch.cuda.current_stream().cuda_stream))


def _buffers(rows, k, l=1):
    """Memory of a quantised operand, as bytes: packed codes, plain scales, scale atoms."""
    return (torch.empty((l, rows, k // 2), dtype=torch.uint8, device="cuda"),
            torch.empty((l, rows, k // 16), dtype=torch.uint8, device="cuda"),
            torch.empty((l, (rows + 127) // 128, k // 64, 32, 4, 4), dtype=torch.uint8, device="cuda"))


def _views(packed, sf, atoms):
    """The operator's views of that memory: [rows, k/2, l], [rows, k/16, l], [32, 4, rest_rows, 4, rest_k, l]."""
    return (packed.permute(1, 2, 0).view(FP4_DTYPE), sf.permute(1, 2, 0).view(SF_DTYPE),
            atoms.permute(3, 4, 1, 5, 2, 0).view(SF_DTYPE))


def _operand(gen, rows, k, l=1):
    """A normally distributed [l][rows][k] tensor, quantised."""
    packed, sf, atoms = _buffers(rows, k, l)
    for i in range(l):
        x = torch.randn((rows, k), dtype=torch.bfloat16, device="cuda", generator=gen).mul_(0.25)
        _quantise(x, packed[i], sf[i], atoms[i])
    return _views(packed, sf, atoms)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, m, k = case["kind"], case["m"], case["k"]
    state = {"kind": kind}
    if kind in ("gemm", "gemv"):
        n, l = case.get("n", 1), case["l"]
        a, sfa, sfa_permuted = _operand(gen, m, k, l)
        b, sfb, sfb_permuted = _operand(gen, n, k, l)
        c = torch.empty((l, m, n), dtype=torch.float16, device="cuda").permute(1, 2, 0)
        state["data"] = (a, b, sfa, sfb, sfa_permuted, sfb_permuted, c)
        return state
    state["x"] = torch.randn((m, k), dtype=torch.bfloat16 if case["bf16"] else torch.float16, device="cuda", generator=gen).mul_(0.25)
    state["quantised"] = _buffers(m, k)
    if kind == "layer":
        n = case["n"]
        a, sfa, sfa_permuted = _views(*state["quantised"])
        b, sfb, sfb_permuted = _operand(gen, n, k)
        state["bias"] = torch.randn(n, dtype=torch.float16, device="cuda", generator=gen)
        state["hidden"] = _buffers(m, n)
        state["hidden_out"] = _views(*state["hidden"])
        state["up"] = (a, b, sfa, sfb, sfa_permuted, sfb_permuted, None)
        h, sfh, sfh_permuted = state["hidden_out"]
        b, sfb, sfb_permuted = _operand(gen, k, n)
        c = torch.empty((1, m, k), dtype=torch.float16, device="cuda").permute(1, 2, 0)
        state["down"] = (h, b, sfh, sfb, sfh_permuted, sfb_permuted, c)
    return state


def run(state):
    kind = state["kind"]
    if kind in ("gemm", "gemv"):
        return custom_kernel(state["data"])
    _quantise(state["x"], *state["quantised"])
    if kind == "quantise":
        return state["quantised"]
    gemm_epilogue(state["up"], bias=state["bias"], activation="silu", nvfp4_out=True, out=state["hidden_out"])
    return custom_kernel(state["down"]), state["hidden"]


def _matmul_bytes(m, n, k, l=1):
    """Operands with their scales, read once, without the output."""
    return l * (m + n) * (k // 2 + k // 16)


def work(case):
    kind, m, k = case["kind"], case["m"], case["k"]
    if kind in ("gemm", "gemv"):
        n, l = case.get("n", 1), case["l"]
        return {"bytes": _matmul_bytes(m, n, k, l) + 2 * l * m * n, "flops": 2 * l * m * n * k}
    quantised = lambda rows, cols: rows * (cols // 2 + 2 * (cols // 16))  # noqa: E731  (codes, and the scales in both layouts)
    if kind == "quantise":
        return {"bytes": 2 * m * k + quantised(m, k), "flops": 4 * m * k}
    # The activations are read once in 16 bits and the result is written once; what lies between is
    # the path's own.  Its two intermediate results are outputs as well.
    n = case["n"]
    return {"bytes": 2 * m * k + 2 * n * (k // 2 + k // 16) + 2 * n + quantised(m, n) + 2 * m * k, "flops": 4 * m * n * k}


def tolerance(case):
    """Quantised operands have so few bits that fp32 sums of their products are all but exact: tile
    shapes, K splits and a recomputation in 64 bits gave the same fp16 values throughout.  What is
    allowed is a value here and there on the other side of a rounding boundary of fp16 (one unit in
    the last place: up to 1e-3 of the value), and where the result is quantised again also of e2m1
    (half a step) or e4m3."""
    if case["kind"] == "quantise":
        return "exact"
    if case["kind"] == "layer":
        return {"rel": 1e-4, "max": 1e-2, "differ": 1e-4}
    return {"rel": 2e-5, "max": 1e-3}

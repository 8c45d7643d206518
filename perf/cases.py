"""Performance cases of the quantised GEMM operators.

Each case is one call (or the two calls that belong together) as a serving program makes it through the package's
public entry points, with its weights, scales and tables already on the GPU.  Four kinds:

``w8a8``     int8 x int8 -> f16 / bf16 with per-token and per-channel scales: single and batched (expert) problems,
             weights as [K, N] or [N, K]; with ``dynamic`` the activations arrive as bf16 / f16 and go through the
             per-token quantiser first, as in a layer whose activations are quantised on the fly.
``grouped``  the ragged form: stacked row groups of different sizes, one expert each.
``w4a16``    f16 / bf16 activations x group-wise int4 weights, one problem or a batch, scalar or per-group zero points.
``w4a8``     bf16 / f16 activations quantised per token x signed int4 weights -> int32 and the token scales.

The fixed sizes are the repository's benchmark configurations and ragged neighbours of them; ``draw`` spreads over the
ranges in between.
"""
import math
import random

import torch

import tilelang_ascend_b200 as q

_DT = {"float16": torch.float16, "bfloat16": torch.bfloat16}


def _w8a8(M, K, N, batch=1, layout="KN", dtype="bfloat16", dynamic=False):
    return {"kind": "w8a8", "batch": batch, "M": M, "K": K, "N": N, "layout": layout, "dtype": dtype, "dynamic": dynamic}


def _grouped(groups, tokens, K, N, dtype="bfloat16", split=1):
    return {"kind": "grouped", "groups": groups, "tokens": tokens, "K": K, "N": N, "dtype": dtype, "split": split}


def _w4a16(M, K, N, batch=1, group=128, dtype="bfloat16", zeros="scalar"):
    return {"kind": "w4a16", "batch": batch, "M": M, "K": K, "N": N, "group": group, "dtype": dtype, "zeros": zeros}


def _w4a8(M, K, N, dtype="bfloat16"):
    return {"kind": "w4a8", "M": M, "K": K, "N": N, "dtype": dtype}


def listed():
    return [
        # a small projection: launch latency and host work decide
        dict(_w8a8(256, 1024, 1024, dtype="float16"), name="w8a8_small"),
        # one decode step of an MLP up-projection for 24 sequences, activations quantised on the fly
        dict(_w8a8(24, 4096, 14336, layout="NK", dynamic=True), name="w8a8_decode"),
        # the same layer's prefill: 4096 tokens
        dict(_w8a8(4096, 4096, 14336, dynamic=True), name="w8a8_prefill"),
        # experts of a mixture with a fixed capacity per expert
        dict(_w8a8(512, 7168, 2048, batch=16), name="w8a8_experts"),
        # the same experts with the tokens as the router dealt them
        dict(_grouped(16, 8192, 7168, 2048), name="w8a8_grouped"),
        # one int4 projection of a decode step, called by itself
        dict(_w4a16(16, 4096, 4096, dtype="float16"), name="w4a16_single"),
        # the same projection for 32 weight sets in one call
        dict(_w4a16(16, 4096, 4096, batch=32, dtype="float16"), name="w4a16_batched"),
        # a large MLP weight at one token: interactive decode
        dict(_w4a16(1, 8192, 28672), name="w4a16_decode_1"),
        # ... at 64 sequences: batched decode
        dict(_w4a16(64, 8192, 28672), name="w4a16_decode_64"),
        # ... a short prompt of ragged length
        dict(_w4a16(500, 8192, 28672), name="w4a16_prompt_500"),
        # ... a long prefill chunk
        dict(_w4a16(4096, 8192, 28672), name="w4a16_prefill_4096"),
        # int8 activations made from bf16 ones, signed int4 weights, decode
        dict(_w4a8(16, 8192, 28672), name="w4a8_decode"),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], uniform in its logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(x / step)) * step))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        dtype = rng.choice(["float16", "bfloat16"])
        kind = rng.choice(["w8a8", "w8a8", "grouped", "w4a16", "w4a16", "w4a16", "w4a16", "w4a8"])
        if kind == "w8a8":
            batch = rng.choice([1, 1, 1, rng.randint(2, 16)])
            dynamic = batch == 1 and rng.random() < 0.5
            case = _w8a8(_log(rng, 1, 4096), _log(rng, 1024, 8192, 32), _log(rng, 1024, 14336, 16), batch,
                         rng.choice(["KN", "NK"]), dtype, dynamic)
        elif kind == "grouped":
            case = _grouped(rng.randint(4, 32), _log(rng, 128, 8192), _log(rng, 1024, 7168, 32),
                            _log(rng, 1024, 4096, 16), dtype, rng.randint(1, 1000000))
        elif kind == "w4a16":
            batch = rng.choice([1, 1, 1, rng.randint(2, 32)])
            M = _log(rng, 1, 4096 if batch == 1 else 64)
            group = rng.choice([128, 128, 128, 128, 64, 256])
            zeros = rng.choice(["scalar", "scalar", "tensor"])
            case = _w4a16(M, _log(rng, 1024, 8192, 256), _log(rng, 1024, 28672 if batch == 1 else 8192, 16), batch,
                          group, dtype, zeros)
        else:
            case = _w4a8(_log(rng, 1, 1024), _log(rng, 1024, 8192, 256), _log(rng, 1024, 28672, 16), dtype)
        if _cost(case) <= most:
            return case


def _sizes(case):
    """Rows of every group, as a router deals them: uneven, none of them empty by design, the sum fixed."""
    rng = random.Random(case["split"])
    w = [rng.uniform(0.2, 1.2) for _ in range(case["groups"])]
    sizes = [int(case["tokens"] * x / sum(w)) for x in w]
    sizes[-1] += case["tokens"] - sum(sizes)
    return tuple(sizes)


def _uniform(shape, lo, hi, gen, dtype=torch.float32):
    return (torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo).to(dtype)


def _int8(shape, gen):
    return torch.randint(-128, 128, shape, generator=gen, device="cuda", dtype=torch.int8)


def _packed(shape, gen):
    return torch.randint(0, 256, shape, generator=gen, device="cuda", dtype=torch.uint8)


def _acts(shape, gen, dtype):
    return torch.randn(shape, generator=gen, device="cuda").to(_DT[dtype])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, K, N = case["kind"], case["K"], case["N"]
    st = {"case": case}
    if kind == "w8a8":
        M, lead = case["M"], (case["batch"],) if case["batch"] > 1 else ()
        st["A"] = _acts((M, K), gen, case["dtype"]) if case["dynamic"] else _int8(lead + (M, K), gen)
        st["B"] = _int8(lead + ((K, N) if case["layout"] == "KN" else (N, K)), gen)
        st["scale"] = _uniform(lead + (N,), 0.001, 0.02, gen)
        if not case["dynamic"]:
            st["scale_a"] = _uniform(lead + (M,), 0.001, 0.02, gen)
        if case["batch"] > 1 and case["layout"] == "KN":
            st["kernel"] = q.simple_quant_batch_matmul(case["batch"], M, N, K, "N", 128, 256, 64, out_dtype=case["dtype"])
    elif kind == "grouped":
        sizes = _sizes(case)
        st["kernel"] = q.grouped_quant_gemm(sizes, K, N, out_dtype=case["dtype"])
        st["meta"] = st["kernel"].block_metadata("cuda")
        st["A"] = _int8((case["tokens"], K), gen)
        st["B"] = _int8((case["groups"], K, N), gen)
        st["scale"] = _uniform((case["groups"], N), 0.001, 0.02, gen)
        st["scale_a"] = _uniform((case["tokens"],), 0.001, 0.02, gen)
    elif kind == "w4a16":
        M, lead, g = case["M"], (case["batch"],) if case["batch"] > 1 else (), case["group"]
        st["A"] = _acts(lead + (M, K), gen, case["dtype"])
        st["B"] = _packed(lead + (N, K // 2), gen)
        st["scales"] = _uniform(lead + (K // g, N), 0.005, 0.02, gen, torch.float16)
        if case["zeros"] == "tensor":
            z = torch.randint(0, 16, lead + (K // g, N), generator=gen, device="cuda")
            st["zeros"], st["mode"] = z.to(torch.float16), "quantized"
        else:
            st["zeros"], st["mode"] = 8, "original"
            if case["batch"] == 1:
                st["kernel"] = q.dequant_gemm_fp16_wrapper(M, N, K, 128, 256, 64, case["dtype"], case["dtype"])
    else:
        M = case["M"]
        st["A"] = _acts((M, K), gen, case["dtype"])
        st["B"] = _packed((N, K // 2), gen)
        st["workspace"] = torch.empty((N, K), dtype=torch.int8, device="cuda")
        st["C"] = torch.empty((M, N), dtype=torch.int32, device="cuda")
        st["kernel"] = q.w4a8_gemm_act_quant(M, N, K) if M <= 128 else q.w4a8_gemm_cv(M, N, K)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "w8a8":
        A, scale_a = st["A"], st.get("scale_a")
        if case["dynamic"]:
            A, scale_a = q.act_quant(A)
            scale_a = scale_a.view(-1)
        if "kernel" in st:
            return st["kernel"](A, st["B"], st["scale"], scale_a)
        return q.quant_matmul(A, st["B"], st["scale"], scale_a=scale_a, out_dtype=case["dtype"], b_layout=case["layout"])
    if kind == "grouped":
        return st["kernel"](st["A"], st["B"], st["meta"], st["scale"], st["scale_a"])
    if kind == "w4a16":
        if "kernel" in st:
            return st["kernel"](st["A"], st["B"], st["scales"], st["zeros"], case["group"])
        return q.w4a16_gemm(st["A"], st["B"], st["scales"], st["zeros"], case["group"], zeros_mode=st["mode"])
    if case["M"] <= 128:
        return st["kernel"](st["A"], st["B"], st["workspace"], st["C"])
    A, scale_a = q.act_quant(st["A"])
    return st["kernel"](A, st["B"], st["workspace"], st["C"]), scale_a.view(-1)


def work(case):
    kind, K, N = case["kind"], case["K"], case["N"]
    if kind == "w8a8":
        b, M = case["batch"], case["M"]
        acts = 2 * M * K if case["dynamic"] else M * K + 4 * M
        return {"bytes": b * (acts + K * N + 4 * N + 2 * M * N), "flops": 2 * b * M * K * N}
    if kind == "grouped":
        used, T = sum(1 for s in _sizes(case) if s), case["tokens"]
        return {"bytes": T * (K + 4 + 2 * N) + used * (K * N + 4 * N), "flops": 2 * T * K * N}
    if kind == "w4a16":
        b, M = case["batch"], case["M"]
        rows = (2 if case["zeros"] == "tensor" else 1) * (K // case["group"])
        return {"bytes": b * (2 * M * K + K * N // 2 + 2 * rows * N + 2 * M * N), "flops": 2 * b * M * K * N}
    M = case["M"]
    return {"bytes": 2 * M * K + K * N // 2 + 4 * M * N + 4 * M, "flops": 2 * M * K * N}


def tolerance(case):
    # int32 sums are exact; the float results are rounded once to the output type (8 or 11 significant bits) after
    # fp32 arithmetic, and the int4 weights of the 16-bit form may carry one f16 rounding of (q - zero) * scale
    if case["kind"] == "w4a8":
        return "exact"
    if case["dtype"] == "bfloat16":
        return {"rel": 5e-3, "max": 2e-2}
    return {"rel": 1e-3, "max": 8e-3}

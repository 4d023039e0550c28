"""The work that a user of the quantized-matmul operators has them do, as measurable cases.

A case is a dict of plain values: the operator (``op``), its sizes and its options.  ``prepare`` makes what a program
holds before the call (weights in the layout they are stored in, scales, activations), ``run`` makes one pass through
the public operators of ``torch_npu`` and returns everything they return.

Operators: ``quant`` (per-token dynamic quantization), ``rms`` (rms_norm), ``rms_quant`` (its fusion with the
quantization), ``w8a8`` (int8 matmul, activations already quantized), ``linear`` (quantization and int8 matmul, the
two calls of one quantized layer), ``w4a16`` (int4 weights, 16-bit activations).
"""
import sys
from pathlib import Path

import torch

_PKG = str(Path(__file__).resolve().parent.parent / "ascend-python_b200")
sys.path.insert(0, _PKG)
try:
    import torch_npu
finally:
    sys.path.remove(_PKG)

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "i8": torch.int8, "i32": torch.int32}


def listed():
    return [
        # one small quantized layer with a batch of 128 tokens: the smallest calls, launches count
        {"name": "linear_small", "op": "linear", "M": 128, "K": 1024, "N": 1024, "dtype": "bf16", "bias": True,
         "trans": False},
        # the input of an 8B-class down projection, a whole prefill batch
        {"name": "quant_prefill", "op": "quant", "M": 8192, "K": 14336, "dtype": "bf16"},
        # normalisation of a ragged batch in half precision
        {"name": "rms_ragged", "op": "rms", "M": 1537, "K": 5120, "dtype": "f16"},
        # normalisation in front of a quantized projection, a whole prefill batch
        {"name": "rms_quant_prefill", "op": "rms_quant", "M": 8192, "K": 4096, "dtype": "bf16"},
        # one token through a 70B-class fused gate/up projection: the weights are streamed once
        {"name": "w8a8_decode_1", "op": "w8a8", "M": 1, "K": 8192, "N": 28672, "dtype": "bf16", "bias": False,
         "trans": False},
        # 32 sequences through a 70B-class down projection: narrow and long
        {"name": "w8a8_decode_32", "op": "w8a8", "M": 32, "K": 28672, "N": 8192, "dtype": "bf16", "bias": True,
         "trans": False},
        # a short ragged prompt through an 8B-class fused QKV projection, weight stored [N, K] as checkpoints have it
        {"name": "w8a8_ragged", "op": "w8a8", "M": 333, "K": 4096, "N": 6144, "dtype": "f16", "bias": True,
         "trans": True},
        # a whole prefill batch through an 8B-class fused gate/up projection
        {"name": "w8a8_prefill", "op": "w8a8", "M": 8192, "K": 4096, "N": 28672, "dtype": "bf16", "bias": False,
         "trans": False},
        # requantized output for an int8 consumer, an 8B-class down projection
        {"name": "w8a8_int8", "op": "w8a8", "M": 2048, "K": 14336, "N": 4096, "dtype": "i8", "bias": True,
         "trans": False},
        # int4 weights, one token
        {"name": "w4a16_decode_1", "op": "w4a16", "M": 1, "K": 8192, "N": 28672, "dtype": "bf16", "group": 128,
         "offset": True, "bias": False},
        # int4 weights, a batch of sequences
        {"name": "w4a16_decode_16", "op": "w4a16", "M": 16, "K": 8192, "N": 28672, "dtype": "bf16", "group": 128,
         "offset": True, "bias": False},
        # int4 weights, a ragged prompt through an 8B-class fused gate/up projection
        {"name": "w4a16_prefill", "op": "w4a16", "M": 1000, "K": 4096, "N": 28672, "dtype": "bf16", "group": 128,
         "offset": True, "bias": True},
    ]


def _log(rng, lo, hi):
    """Uniform over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(["linear", "quant", "rms", "rms_quant", "w8a8", "w8a8", "w8a8", "w4a16", "w4a16", "w4a16"])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    if op in ("quant", "rms", "rms_quant"):
        # hidden sizes are multiples of eight; one in six is odd
        cols = _log(rng, 512, 16384)
        cols = cols | 1 if rng.random() < 1 / 6 else cols // 8 * 8
        return {"op": op, "M": _log(rng, 1, 8192), "K": cols, "dtype": dtype}
    if op == "w4a16":
        K, N = 128 * _log(rng, 8, 224), 8 * _log(rng, 128, 3584)
        M = _log(rng, 1, 2048)
        while M * K * N > 1000 * 4096 * 28672:
            M = M // 2 + (M // 2) % 2
        return {"op": op, "M": M, "K": K, "N": N, "dtype": dtype, "group": rng.choice([128, 128, 128, 0]),
                "offset": rng.random() < 0.7, "bias": rng.random() < 0.3}
    trans = rng.random() < 0.4
    K, N = 16 * _log(rng, 64, 1792), 16 * _log(rng, 64, 1792)
    if trans and rng.random() < 0.3:
        N += rng.randrange(1, 16)  # any number of columns goes with weights stored [N, K]
    M = _log(rng, 1, 8192)
    while M * K * N > 8192 * 4096 * 28672 // 2:
        M = M // 2 + (M // 2) % 2
    if op == "w8a8":
        dtype = rng.choice(["bf16", "bf16", "f16", "i8", "i32"])
    return {"op": op, "M": M, "K": K, "N": N, "dtype": dtype, "bias": rng.random() < 0.5, "trans": trans}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op, M, K = case["op"], case["M"], case["K"]
    dtype = _DTYPES[case["dtype"]]
    real = dtype if dtype.is_floating_point else torch.bfloat16

    def normal(*shape, std=1.0, to=real):
        return (torch.randn(shape, generator=g, device="cuda") * std).to(to)

    def uniform(n, lo, hi, to=torch.float32):
        return (torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo).to(to)

    s = {"op": op, "dtype": dtype, "x": normal(M, K)}
    if op in ("rms", "rms_quant"):
        s["gamma"] = uniform(K, 0.5, 1.5, to=real)
    if op == "w4a16":
        N, group = case["N"], case["group"]
        rows = K // (group or K)
        s["weight"] = torch.randint(-2**31, 2**31, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
        s["scale"] = uniform((rows, N), 5e-3, 2e-2, to=real)
        s["offset"] = uniform((rows, N), -1.0, 1.0, to=real) if case["offset"] else None
        s["bias"] = normal(N, std=0.1) if case["bias"] else None
        s["group"] = group
    if op in ("w8a8", "linear"):
        N = case["N"]
        shape = (N, K) if case["trans"] else (K, N)
        weight = torch.randint(-127, 128, shape, generator=g, device="cuda", dtype=torch.int8)
        s["weight"] = weight.t() if case["trans"] else weight
        s["scale"] = uniform(N, 1e-3, 1e-2)
        s["bias"], s["offset"] = None, None
        if case["bias"]:
            s["bias"] = (normal(N, std=0.1) if dtype.is_floating_point else
                         torch.randint(-4096, 4096, (N,), generator=g, device="cuda", dtype=torch.int32))
    if op == "w8a8":
        x = s.pop("x").float()
        pertoken = x.abs().amax(dim=1) / 127.0
        s["x"] = torch.round(x / pertoken[:, None]).to(torch.int8)
        s["pertoken"] = pertoken if dtype != torch.int32 else None
        if dtype == torch.int8:
            # an output that spans the int8 range: x has unit variance, the weights a deviation of about 73
            s["scale"] = uniform(N, 0.5, 1.5) * (40.0 / (73.0 * K**0.5))
            s["offset"] = uniform(N, -8.0, 8.0)
    return s


def run(s):
    op, x = s["op"], s["x"]
    if op == "quant":
        return torch_npu.npu_dynamic_quant(x)
    if op == "rms":
        return torch_npu.npu_rms_norm(x, s["gamma"])
    if op == "rms_quant":
        return torch_npu.npu_rms_norm_dynamic_quant(x, s["gamma"])
    if op == "w4a16":
        return torch_npu.npu_weight_quant_batchmatmul(x, s["weight"], s["scale"], s["offset"], bias=s["bias"],
                                                      antiquant_group_size=s["group"])
    if op == "linear":
        q, pertoken = torch_npu.npu_dynamic_quant(x)
        y = torch_npu.npu_quant_matmul(q, s["weight"], s["scale"], pertoken_scale=pertoken, bias=s["bias"],
                                       output_dtype=s["dtype"])
        return q, pertoken, y
    return torch_npu.npu_quant_matmul(x, s["weight"], s["scale"], offset=s["offset"], pertoken_scale=s["pertoken"],
                                      bias=s["bias"], output_dtype=s["dtype"])


def work(case):
    op, M, K = case["op"], case["M"], case["K"]
    if op == "quant":
        return {"bytes": 3 * M * K + 4 * M, "flops": 4 * M * K}
    if op == "rms":
        return {"bytes": 4 * M * K + 4 * M + 2 * K, "flops": 4 * M * K}
    if op == "rms_quant":
        return {"bytes": 3 * M * K + 8 * M + 2 * K, "flops": 8 * M * K}
    N = case["N"]
    flops = 2 * M * N * K
    if op == "w4a16":
        table = 2 * (K // (case["group"] or K)) * N
        return {"bytes": K * N // 2 + table * (2 if case["offset"] else 1) + 2 * M * K + 2 * M * N +
                (2 * N if case["bias"] else 0), "flops": flops}
    out = {"bf16": 2, "f16": 2, "i8": 1, "i32": 4}[case["dtype"]]
    rest = 4 * N * (2 if case["dtype"] == "i8" else 1) + 4 * M + (out * N if case["bias"] else 0)
    x = 2 * M * K + M * K if op == "linear" else M * K  # the quantized activations are one of its outputs
    return {"bytes": x + K * N + out * M * N + rest, "flops": flops}


def tolerance(case):
    """What another correct implementation of the same precision may differ by, each about four times what comparing
    the operators with 64 bits (or with their sums in another order) shows."""
    op, dtype = case["op"], case["dtype"]
    if op == "quant":
        return "exact"  # IEEE divisions of a maximum: nothing depends on an order
    if op in ("linear", "w8a8"):
        if dtype in ("i8", "i32"):
            return "exact"
        # exact integer sums; the product of the two scales may round differently, which moves some results by one unit
        return {"rel": 4e-4, "max": 8e-3} if dtype == "bf16" else {"rel": 6e-5, "max": 1e-3}
    if op == "rms":
        return {"rel": 2e-4, "max": 8e-3} if dtype == "bf16" else {"rel": 5e-5, "max": 1e-3}
    if op == "rms_quant":
        # the sum of squares in another order moves some normalised values by one unit, and with them a few integers,
        # or, where the moved value is the row's largest, that row's scale
        return {"rel": 2e-3, "max": 5e-2, "differ": 2e-2} if dtype == "bf16" else {"rel": 1e-3, "max": 3e-2, "differ": 2e-2}
    # 16-bit weights and outputs, sums of thousands of rounded products
    return {"rel": 1e-2, "max": 8e-2} if dtype == "bf16" else {"rel": 1.5e-3, "max": 1e-2}


def exact(case, seed):
    s = prepare(case, seed)
    op, x = s["op"], s["x"].double()

    def quantize(v):
        scale = v.abs().amax(dim=1) / 127.0
        return torch.round(v / scale[:, None]).clamp(-128, 127).to(torch.int8), scale

    if op == "quant":
        return quantize(x)
    if op in ("rms", "rms_quant"):
        rstd = 1.0 / torch.sqrt(x.square().mean(dim=1, keepdim=True) + 1e-6)
        y = x * rstd * s["gamma"].double()
        if op == "rms":
            return y, rstd
        return (*quantize(y.to(s["x"].dtype).double()), rstd)  # the quantization is that of the 16-bit values
    if op == "w4a16":
        K = x.shape[1]
        group = s["group"] or K
        y = torch.zeros(x.shape[0], s["scale"].shape[1], dtype=torch.float64, device="cuda")
        shifts = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
        step = min(group, 1024)
        for k in range(0, K, step):
            rows = s["weight"][k:k + step]
            w = ((rows[:, :, None] >> shifts) & 15).reshape(rows.shape[0], -1)
            w = torch.where(w > 7, w - 16, w).double()
            if s["offset"] is not None:
                w += s["offset"][k // group].double()
            y += x[:, k:k + step] @ (w * s["scale"][k // group].double())
        return y if s["bias"] is None else y + s["bias"].double()
    q, pertoken = (s["x"], s["pertoken"]) if op == "w8a8" else quantize(x)
    y = q.double() @ s["weight"].double()
    whole = not s["dtype"].is_floating_point
    if whole and s["bias"] is not None:
        y += s["bias"]
    if s["dtype"] == torch.int32:
        return y.to(torch.int32)
    y = y * s["scale"].double() * pertoken.double()[:, None]
    if whole:
        return torch.round(y + s["offset"].double()).clamp(-128, 127).to(torch.int8)
    if s["bias"] is not None:
        y += s["bias"].double()
    return (q, pertoken, y) if op == "linear" else y

"""What a user of this library has it do, as timed cases: quantized-matmul calls of an inference
program over the range of sizes, batches, formats and options that the entry points serve.

Seven kinds of work, each through the public entry points:

  layer      one decode step through a decoder layer's projections (q + k + v fused, output
             projection, up + gate with the activation, down), one token, GGUF blocks
  gemm       batched decode on one prepared matrix: f32 activations, 1 to 32 rows, GGUF blocks
  host       the drop-in call on host buffers (activations in, results out, synchronous)
  prefill    bf16 prompt tokens against one prepared GGUF matrix
  w8a8       int8 weights x int8 activations, symmetric and with activation zero points
  canonical  prepared checkpoint tensors (SmoothQuant int8 with channel scales, AWQ / GPTQ uint4
             and symmetric int4 with group scales), typed input and output, bias, activation
  w4a8       compact int4 rows x activations quantized to int8 on the fly
"""

from __future__ import annotations

import numpy as np
import torch

import __graft_entry__

qx = __graft_entry__.load_package()

Q8_0, Q4_0 = qx.Q8_0, qx.Q4_0
FORMATS = {"q8_0": Q8_0, "q4_0": Q4_0}
TYPES = {"f32": (qx.F32, torch.float32), "f16": (qx.F16, torch.float16),
         "bf16": (qx.BF16, torch.bfloat16)}
ACTIVATIONS = {"none": qx.ACT_NONE, "gelu_erf": qx.ACT_GELU_ERF, "gelu_tanh": qx.ACT_GELU_TANH,
               "silu": qx.ACT_SILU, "relu2": qx.ACT_RELU2}


def listed():
    return [
        # the smallest call that a program ported from the CPU library makes: one token, host
        # buffers on both sides, so that launches, copies and the synchronisation are what counts
        dict(name="host_q8_0_4096x4096", kind="host", fmt="q8_0", m=1, n=4096, k=4096),
        # one decode step of a chat session: every projection of a decoder layer, one token
        dict(name="layer_q4_0_4096_14336", kind="layer", fmt="q4_0", hidden=4096, kv=1024, ffn=14336),
        # a few sessions decoded together (or a speculated run of tokens) on 4-bit blocks
        dict(name="gemm_q4_0_m8_14336x4096", kind="gemm", fmt="q4_0", m=8, n=14336, k=4096),
        # the largest decode batch of one launch on the largest 8-bit matrix
        dict(name="gemm_q8_0_m32_28672x8192", kind="gemm", fmt="q8_0", m=32, n=28672, k=8192),
        # a long prompt on the largest 4-bit matrix: the tensor-bound end of the range
        dict(name="prefill_q4_0_m2048_28672x8192", kind="prefill", fmt="q4_0", m=2048, n=28672, k=8192),
        # a prompt of an arbitrary length on 8-bit blocks, down projection
        dict(name="prefill_q8_0_m331_4096x11008", kind="prefill", fmt="q8_0", m=331, n=4096, k=11008),
        # prefill of a W8A8 checkpoint
        dict(name="w8a8_m512_14336x4096", kind="w8a8", m=512, n=14336, k=4096, azp=False),
        # decode-sized W8A8 with activation zero points: a call of a few microseconds
        dict(name="w8a8_azp_m4_1024x1408", kind="w8a8", m=4, n=1024, k=1408, azp=True),
        # one decoded token on a SmoothQuant checkpoint used weight-only, whole epilogue
        dict(name="canonical_int8_m1_14336x4096", kind="canonical", layout="int8", group=0, m=1,
             n=14336, k=4096, x_type="bf16", y_type="bf16", bias=True, activation="silu"),
        # batched decode on an AWQ / GPTQ checkpoint
        dict(name="canonical_u4_m16_14336x4096", kind="canonical", layout="uint4", group=128, m=16,
             n=14336, k=4096, x_type="f16", y_type="f16", bias=False, activation="none"),
        # a prompt on an AWQ / GPTQ checkpoint
        dict(name="canonical_u4_m512_14336x4096", kind="canonical", layout="uint4", group=128, m=512,
             n=14336, k=4096, x_type="bf16", y_type="bf16", bias=True, activation="none"),
        # batched decode on compact int4 rows with dynamic int8 activations
        dict(name="w4a8_m16_4096x4096", kind="w4a8", m=16, n=4096, k=4096),
    ]


def _spread(rng, low, high, step=1):
    """Log-uniform over [low, high], a multiple of `step`."""
    value = low * (high / low) ** rng.random()
    return max(step, int(round(value / step)) * step)


def draw(rng):
    kind = rng.choice(("layer", "gemm", "host", "prefill", "w8a8", "canonical", "canonical", "w4a8"))
    if kind == "layer":
        hidden = _spread(rng, 1024, 6144, 128)
        return dict(kind=kind, fmt=rng.choice(("q8_0", "q4_0")), hidden=hidden,
                    kv=max(128, hidden // rng.choice((1, 4, 8)) // 128 * 128),
                    ffn=_spread(rng, 2 * hidden, 4 * hidden, 32))
    if kind == "gemm":
        return dict(kind=kind, fmt=rng.choice(("q8_0", "q4_0")), m=_spread(rng, 1, 32),
                    n=_spread(rng, 512, 28672), k=_spread(rng, 512, 8192, 32))
    if kind == "host":
        return dict(kind=kind, fmt=rng.choice(("q8_0", "q4_0")), m=_spread(rng, 1, 32),
                    n=_spread(rng, 512, 14336), k=_spread(rng, 512, 8192, 32))
    if kind == "prefill":
        return dict(kind=kind, fmt=rng.choice(("q8_0", "q4_0")), m=_spread(rng, 64, 1536),
                    n=_spread(rng, 1024, 14336), k=_spread(rng, 1024, 8192, 32))
    if kind == "w8a8":
        return dict(kind=kind, m=_spread(rng, 1, 2048), n=_spread(rng, 1024, 14336),
                    k=_spread(rng, 1024, 8192, rng.choice((16, 128))), azp=rng.random() < 0.4)
    if kind == "canonical":
        layout = rng.choice(("int8", "uint4", "uint4", "int4"))
        group = 0 if layout == "int8" else rng.choice((32, 64, 128, 128))
        return dict(kind=kind, layout=layout, group=group, m=_spread(rng, 1, 1024),
                    n=_spread(rng, 1024, 14336), k=_spread(rng, 1024, 8192, group or 16),
                    x_type=rng.choice(("bf16", "bf16", "f16", "f32")),
                    y_type=rng.choice(("bf16", "bf16", "f16", "f32")), bias=rng.random() < 0.5,
                    activation=rng.choice(("none", "none", "silu", "gelu_tanh", "gelu_erf", "relu2")))
    return dict(kind=kind, m=_spread(rng, 1, 64), n=_spread(rng, 1024, 14336),
                k=_spread(rng, 1024, 8192, 2))


# ---- inputs -----------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, count, low, high):
    return torch.rand(count, generator=g, device="cuda") * (high - low) + low


def _codes(g, count, low, high, dtype):
    return torch.randint(low, high, (count,), generator=g, device="cuda", dtype=torch.int32).to(dtype)


def _blocks(g, fmt, n, k, low, high):
    """GGUF blocks on the device: an fp16 scale of magnitude [low, high) and either sign, then
    32 int8 codes (q8_0) or 16 bytes of nibbles (q4_0)."""
    blocks = n * (k // 32)
    code_bytes = 32 if fmt == Q8_0 else 16
    scale = _uniform(g, blocks, low, high) * (_codes(g, blocks, 0, 2, torch.float32) * 2 - 1)
    out = torch.empty((blocks, 2 + code_bytes), dtype=torch.uint8, device="cuda")
    out[:, :2] = scale.half().view(torch.uint8).view(blocks, 2)
    codes = torch.randint(0, 256, (blocks, code_bytes), generator=g, device="cuda", dtype=torch.uint8)
    if fmt == Q8_0:
        codes[codes == 128] = 127  # quantizers emit -127 .. 127
    out[:, 2:] = codes
    return out.view(-1)


SCALES = {Q8_0: (0.001, 0.02), Q4_0: (0.002, 0.04)}


def _layer_scale(fmt, k):
    """Scales that keep a projection's outputs at the size of its inputs."""
    rms = (73.3 if fmt == Q8_0 else 4.6) * k ** 0.5
    return 0.5 / rms, 1.5 / rms


def _prepared(fmt, packed, n, k):
    weights = qx.PackedWeights()
    qx.check(weights.prepare(fmt, packed, n, k), "prepare")
    return weights


def _fused(fmt, parts, rows, k):
    weights = qx.PackedWeights()
    qx.check(weights.prepare_fused(fmt, [p.cpu().numpy() for p in parts], rows, k), "prepare_fused")
    weights._fused_keepalive = None  # the handle holds its own copy
    return weights


def _w8a8_inputs(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    w = _codes(g, n * k, -127, 128, torch.int8).view(n, k)
    state = dict(kind="w8a8", azp=case["azp"], m=m, n=n, k=k, w=w,
                 x=_codes(g, m * k, -127, 128, torch.int8).view(m, k),
                 ws=_uniform(g, n, 0.001, 0.01), xs=_uniform(g, m, 0.005, 0.05))
    if case["azp"]:
        state["row_sum"] = w.sum(dim=1, dtype=torch.int32)
        state["zp"] = _codes(g, m, -20, 21, torch.int32)
    return state


def _canonical_inputs(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    groups = k // case["group"] if case["group"] else 1
    level = 73.3 if case["layout"] == "int8" else 4.6
    scales = _uniform(g, n * groups, 0.5, 1.5) / (level * k ** 0.5)
    if case["layout"] == "int8":
        data = _codes(g, n * k, -127, 128, torch.int8).view(torch.uint8)
    else:
        data = torch.randint(0, 256, (n * k // 2,), generator=g, device="cuda", dtype=torch.uint8)
    zeros = _codes(g, n * groups, 5, 11, torch.float32) if case["layout"] == "uint4" else None
    x = torch.randn((m, k), generator=g, device="cuda").to(TYPES[case["x_type"]][1])
    bias = torch.randn(n, generator=g, device="cuda") * 0.1 if case["bias"] else None
    return data, scales, zeros, x, bias


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "layer":
        fmt, h, kv, ffn = FORMATS[case["fmt"]], case["hidden"], case["kv"], case["ffn"]
        over_h, over_f = _layer_scale(fmt, h), _layer_scale(fmt, ffn)
        qkv = _fused(fmt, [_blocks(g, fmt, n, h, *over_h) for n in (h, kv, kv)], [h, kv, kv], h)
        up_gate = _fused(fmt, [_blocks(g, fmt, ffn, h, *over_h) for _ in range(2)], [ffn, ffn], h)
        return dict(kind=kind, qkv=qkv, up_gate=up_gate,
                    o=_prepared(fmt, _blocks(g, fmt, h, h, *over_h), h, h),
                    down=_prepared(fmt, _blocks(g, fmt, h, ffn, *over_f), h, ffn),
                    x=torch.randn((1, h), generator=g, device="cuda"),
                    q=torch.zeros((1, h), device="cuda"), k=torch.zeros((1, kv), device="cuda"),
                    v=torch.zeros((1, kv), device="cuda"), a=torch.zeros((1, h), device="cuda"),
                    mid=torch.zeros(ffn, device="cuda"), both=torch.zeros(2 * ffn, device="cuda"),
                    y=torch.zeros((1, h), device="cuda"))
    m, n, k = case["m"], case["n"], case["k"]
    if kind in ("gemm", "host", "prefill"):
        fmt = FORMATS[case["fmt"]]
        weights = _prepared(fmt, _blocks(g, fmt, n, k, *SCALES[fmt]), n, k)
        x = torch.randn((m, k), generator=g, device="cuda")
        if kind == "host":
            return dict(kind=kind, weights=weights, m=m, x=x.cpu().numpy(),
                        y=np.zeros((m, n), np.float32))
        if kind == "prefill":
            x = x.bfloat16().view(torch.int16)
        return dict(kind=kind, weights=weights, m=m, x=x, y=torch.zeros((m, n), device="cuda"))
    if kind == "w8a8":
        return dict(_w8a8_inputs(case, g), y=torch.zeros((m, n), device="cuda"))
    if kind == "canonical":
        layout = {"int8": qx.INT8_SYMMETRIC, "uint4": qx.UINT4_AFFINE, "int4": qx.INT4_SYMMETRIC}[case["layout"]]
        data, scales, zeros, x, bias = _canonical_inputs(case, g)
        # (host arrays of its own: a view points into them)
        host = (data.cpu().numpy(), scales.cpu().numpy())
        zeros = None if zeros is None else zeros.cpu().numpy()
        mode = qx.SCALE_GROUP if case["group"] else qx.SCALE_CHANNEL
        weights = qx.CanonicalWeights()
        qx.check(weights.prepare(qx.canonical_view(layout, mode, n, k, case["group"] or k, *host, zeros=zeros)),
                 "prepare")
        x_type = TYPES[case["x_type"]][0]
        y_type, y_torch = TYPES[case["y_type"]]
        return dict(kind=kind, weights=weights, m=m, x_type=x_type, y_type=y_type,
                    x=x, y=torch.zeros((m, n), device="cuda", dtype=y_torch), bias=bias,
                    activation=ACTIVATIONS[case["activation"]])
    packed = torch.randint(0, 256, (n * k // 2,), generator=g, device="cuda", dtype=torch.uint8)
    return dict(kind=kind, m=m, n=n, k=k, packed=packed,
                scales=_uniform(g, n, 0.5, 1.5) / (4.6 * k ** 0.5),
                x=torch.randn((m, k), generator=g, device="cuda"),
                y=torch.zeros((m, n), device="cuda"),
                scratch=torch.empty(int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)), dtype=torch.uint8,
                                    device="cuda"))


def run(state):
    kind = state["kind"]
    if kind == "layer":
        s = state
        qx.check(s["qkv"].qgemm_fused_dev(s["x"], [s["q"], s["k"], s["v"]], 1), "qkv")
        # (attention is the caller's: the query projection stands in for its output)
        qx.check(s["o"].qgemm_dev(s["q"], s["a"], 1), "o")
        qx.check(s["up_gate"].up_gate_activation_dev(s["a"], s["mid"], s["both"], False), "up_gate")
        qx.check(s["down"].qgemm_dev(s["mid"], s["y"], 1), "down")
        return s["q"], s["k"], s["v"], s["mid"], s["y"]
    if kind == "gemm":
        qx.check(state["weights"].qgemm_dev(state["x"], state["y"], state["m"]), "qgemm")
    elif kind == "host":
        qx.check(state["weights"].qgemm_prepacked(state["x"], state["m"], state["y"])[0], "qgemm_prepacked")
    elif kind == "prefill":
        qx.check(state["weights"].qgemm_bf16_dev(state["x"], state["y"], state["m"]), "qgemm_bf16")
    elif kind == "w8a8":
        qx.check(qx.int8_gemm_dev(state["w"], state["x"], state["ws"], state["xs"], state["y"], state["m"],
                                  state["n"], state["k"], row_sum=state.get("row_sum"), zp=state.get("zp")),
                 "int8_gemm")
    elif kind == "canonical":
        qx.check(state["weights"].qgemm_storage_dev(state["x"], state["x_type"], state["y"], state["y_type"],
                                                    state["m"], bias=state["bias"],
                                                    activation=state["activation"]), "qgemm_storage")
    else:
        qx.check(qx.lib.qx_lowbit_gemm_w8a8_dev(
            state["packed"].data_ptr(), state["scales"].data_ptr(), state["x"].data_ptr(),
            state["y"].data_ptr(), state["scratch"].data_ptr(), state["m"], state["n"], state["k"],
            torch.cuda.current_stream().cuda_stream), "lowbit_gemm_w8a8")
    return state["y"]


# ---- what a pass cannot do without ------------------------------------------------------------

def _block_matrix_bytes(fmt, n, k):
    return n * (k // 32) * (34 if fmt == "q8_0" else 18)


def work(case):
    kind = case["kind"]
    if kind == "layer":
        h, kv, ffn = case["hidden"], case["kv"], case["ffn"]
        shapes = ((h + 2 * kv, h), (h, h), (2 * ffn, h), (h, ffn))
        weights = sum(_block_matrix_bytes(case["fmt"], n, k) for n, k in shapes)
        return {"bytes": weights + 4 * (h + h + 2 * kv + ffn + h),
                "flops": 2 * sum(n * k for n, k in shapes)}
    m, n, k = case["m"], case["n"], case["k"]
    flops = 2 * m * n * k
    if kind in ("gemm", "host"):
        return {"bytes": _block_matrix_bytes(case["fmt"], n, k) + 4 * m * (n + k), "flops": flops}
    if kind == "prefill":
        return {"bytes": _block_matrix_bytes(case["fmt"], n, k) + 2 * m * k + 4 * m * n, "flops": flops}
    if kind == "w8a8":
        return {"bytes": n * k + m * k + 4 * m * n + 4 * (m + n) * (2 if case["azp"] else 1), "flops": flops}
    if kind == "canonical":
        groups = k // case["group"] if case["group"] else 1
        size = {"f32": 4, "f16": 2, "bf16": 2}
        tables = n * groups * (8 if case["layout"] == "uint4" else 4) + (4 * n if case["bias"] else 0)
        return {"bytes": n * k // (1 if case["layout"] == "int8" else 2) + tables +
                m * k * size[case["x_type"]] + m * n * size[case["y_type"]], "flops": flops}
    return {"bytes": n * k // 2 + 4 * n + 4 * m * (n + k), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("w8a8", "w4a8"):
        return "exact"  # exact integer sums, then the same two rounded multiplies
    # Against the same product in float64: f32 outputs are 1e-7 to 8e-7 off (5e-6 at the largest
    # difference, behind an activation), the q4_0 prefill 1.8e-4 (1.1e-3), typed outputs move by
    # one unit of their type in one value of 1e3 to 1e4.
    if kind == "prefill" and case["fmt"] == "q4_0":
        return {"rel": 7e-4, "max": 5e-3}  # fp16 weights: one rounding of d * (nibble - 8) each
    if kind == "canonical" and case["y_type"] != "f32":
        return {"rel": 5e-4, "max": 1e-2} if case["y_type"] == "bf16" else {"rel": 6e-5, "max": 1.3e-3}
    return {"rel": 4e-6, "max": 4e-5}  # 32-bit sums


# ---- the same values in 64 bits ---------------------------------------------------------------

def _dense_blocks(fmt, blocks, n, k):
    b = blocks.view(n, k // 32, -1)
    d = b[..., :2].contiguous().view(torch.float16).double()
    if fmt == Q8_0:
        codes = b[..., 2:].contiguous().view(torch.int8).double()
    else:
        codes = torch.cat((b[..., 2:] & 15, b[..., 2:] >> 4), dim=-1).double() - 8.0
    return (d * codes).view(n, k)


def _dense_nibbles(packed, n, k):
    b = packed.view(n, k // 2)
    return torch.stack((b & 15, b >> 4), dim=-1).view(n, k).double()


def _activate(v, activation):
    if activation == "gelu_erf":
        return torch.nn.functional.gelu(v)
    if activation == "gelu_tanh":
        return torch.nn.functional.gelu(v, approximate="tanh")
    if activation == "silu":
        return torch.nn.functional.silu(v)
    return torch.relu(v) ** 2 if activation == "relu2" else v


def exact(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "layer":  # the draws of prepare(), in its order
        fmt, h, kv, ffn = FORMATS[case["fmt"]], case["hidden"], case["kv"], case["ffn"]
        over_h, over_f = _layer_scale(fmt, h), _layer_scale(fmt, ffn)
        wq, wk, wv = (_dense_blocks(fmt, _blocks(g, fmt, n, h, *over_h), n, h) for n in (h, kv, kv))
        up, gate = (_dense_blocks(fmt, _blocks(g, fmt, ffn, h, *over_h), ffn, h) for _ in range(2))
        wo = _dense_blocks(fmt, _blocks(g, fmt, h, h, *over_h), h, h)
        down = _dense_blocks(fmt, _blocks(g, fmt, h, ffn, *over_f), h, ffn)
        x = torch.randn((1, h), generator=g, device="cuda").double()
        q, key, value = x @ wq.T, x @ wk.T, x @ wv.T
        a = q @ wo.T
        mid = torch.nn.functional.silu(a @ gate.T) * (a @ up.T)
        return q, key, value, mid[0], mid @ down.T
    m, n, k = case["m"], case["n"], case["k"]
    if kind in ("gemm", "host", "prefill"):
        fmt = FORMATS[case["fmt"]]
        w = _dense_blocks(fmt, _blocks(g, fmt, n, k, *SCALES[fmt]), n, k)
        x = torch.randn((m, k), generator=g, device="cuda")
        y = (x.bfloat16() if kind == "prefill" else x).double() @ w.T
        return y.cpu().numpy() if kind == "host" else y
    if kind == "w8a8":
        s = _w8a8_inputs(case, g)
        acc = s["x"].double() @ s["w"].double().T
        if case["azp"]:
            acc -= s["zp"].double()[:, None] * s["row_sum"].double()[None, :]
        return acc * s["ws"].double()[None, :] * s["xs"].double()[:, None]
    if kind == "canonical":
        data, scales, zeros, x, bias = _canonical_inputs(case, g)
        w = data.view(torch.int8).view(n, k).double() if case["layout"] == "int8" else _dense_nibbles(data, n, k)
        if case["layout"] == "int4":
            w = torch.where(w >= 8, w - 16, w)
        w = w.view(n, scales.numel() // n, -1)
        if zeros is not None:
            w = w - zeros.double().view(n, -1, 1)
        w = (w * scales.double().view(n, -1, 1)).view(n, k)
        y = x.double() @ w.T
        return _activate(y if bias is None else y + bias.double(), case["activation"])
    packed = torch.randint(0, 256, (n * k // 2,), generator=g, device="cuda", dtype=torch.uint8)
    ws = _uniform(g, n, 0.5, 1.5) / (4.6 * k ** 0.5)
    x = torch.randn((m, k), generator=g, device="cuda")
    # the int8 activation codes are part of the operation: one scale per token, rounded in 32 bits
    xs = x.abs().amax(dim=1, keepdim=True) / 127.0
    codes = torch.round(x * (1.0 / xs)).clamp(-127, 127)
    acc = codes.double() @ (_dense_nibbles(packed, n, k) - 8.0).T
    return acc * ws.double()[None, :] * xs.double()

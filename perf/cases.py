"""The work that a serving program has this package do, as timed cases.

Every case goes through the public entry points of ``metal_native``.  Sizes are those of the
repository's benchmark configurations (the MLP projections of Qwen2.5-0.5B / 7B, Llama-3-8B / 70B) or
generic; ``draw`` spreads over the same ranges.  Weights are loaded once and served, so the
program declares them immutable, as ``bench.py`` does.

Kinds of case
  linear      one projection, ``dequant_matmul`` called as the reference's binding is (the result is
              allocated by the call), or ``dequant_matmul_fused`` where an epilogue is asked for
  step        one MLP block of a decode step -- residual add + RMSNorm, gate+up with SwiGLU (fused where
              ``dequant_matmul_swiglu`` takes the batch, else applied by torch), down with the residual
              added -- recorded by ``PhasePipeline.capture_step`` and replayed
  host        one projection with activations and result in pinned host memory, waited for
  dequantize  a whole weight matrix to 16 bits: ``dequantize`` (scale and zero) or ``dequantize_flat``
  norm        ``fused_residual_norm`` of a block of rows, with the new residual stream stored
"""
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "metal-native_b200"))

import metal_native  # noqa: E402

C = metal_native._C
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}

# The most a drawn case may cost: the largest listed ones.
MAX_MACS = 4096 * 4096 * 14336
MAX_WEIGHTS = 8192 * 57344


def listed():
    return [
        # the smallest call a decode loop makes: one token through the down projection of a 0.5B model; launch latency
        {"name": "linear_m1_small", "kind": "linear", "m": 1, "k": 4864, "n": 896, "quant": "int4", "group": 64,
         "dtype": "fp16", "zeros": True, "epilogue": "none"},
        # single-stream decode of a 7B model: the whole MLP block of one token
        {"name": "step_m1_7b", "kind": "step", "m": 1, "k": 3584, "h": 18944, "quant": "int4", "group": 128,
         "dtype": "fp16", "zeros": True},
        # sixteen sequences decoded together on an 8B model, bf16 and symmetric
        {"name": "step_m16_8b", "kind": "step", "m": 16, "k": 4096, "h": 14336, "quant": "int4", "group": 128,
         "dtype": "bf16", "zeros": False},
        # a server's decode batch on the largest layer: 70B gate+up, int8 with one scale per row, 64 sequences
        {"name": "linear_m64_70b_int8", "kind": "linear", "m": 64, "k": 8192, "n": 57344, "quant": "int8", "group": 8192,
         "dtype": "bf16", "zeros": False, "epilogue": "none"},
        # a middling decode batch with int8 groups of 64
        {"name": "linear_m24_int8_g64", "kind": "linear", "m": 24, "k": 4096, "n": 6144, "quant": "int8", "group": 64,
         "dtype": "fp16", "zeros": True, "epilogue": "none"},
        # prefill of a 512-token prompt on a 7B model: the wide projection ...
        {"name": "prefill_m512_up", "kind": "linear", "m": 512, "k": 3584, "n": 18944, "quant": "int4", "group": 128,
         "dtype": "fp16", "zeros": True, "epilogue": "none"},
        # ... and the narrow, long one
        {"name": "prefill_m512_down", "kind": "linear", "m": 512, "k": 18944, "n": 3584, "quant": "int4", "group": 128,
         "dtype": "fp16", "zeros": True, "epilogue": "none"},
        # prefill of a long prompt (or of several) on an 8B model in bf16
        {"name": "prefill_m4096_bf16", "kind": "linear", "m": 4096, "k": 4096, "n": 14336, "quant": "int4", "group": 128,
         "dtype": "bf16", "zeros": False, "epilogue": "none"},
        # an odd prompt length, an odd number of columns, the smallest group size, and an epilogue
        {"name": "ragged_m197_g32", "kind": "linear", "m": 197, "k": 4160, "n": 5003, "quant": "int4", "group": 32,
         "dtype": "fp16", "zeros": True, "epilogue": "bias_silu"},
        # a caller that keeps activations and results in host memory
        {"name": "host_m1_7b", "kind": "host", "m": 1, "k": 3584, "n": 18944, "quant": "int4", "group": 128,
         "dtype": "fp16", "zeros": True},
        # a layer expanded once for a caller that wants plain fp16 weights
        {"name": "dequantize_7b", "kind": "dequantize", "k": 3584, "n": 18944, "quant": "int4", "group": 128,
         "dtype": "fp16", "zeros": True, "flat": False},
        # the normalisation in front of a prefill's MLP
        {"name": "norm_8192x4096", "kind": "norm", "m": 8192, "k": 4096, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choices(["linear", "step", "host", "dequantize", "norm"], [60, 20, 4, 8, 8])[0]
    dtype = rng.choice(["fp16", "bf16"])
    if kind == "norm":
        m = _log(rng, 1, 8192)
        k = 8 * _log(rng, 112, 1024) if rng.random() < 0.8 else _log(rng, 900, 8191)
        return {"kind": kind, "m": m, "k": k, "dtype": dtype}
    quant = rng.choices(["int4", "int8"], [65, 35])[0]
    k = 64 * _log(rng, 14, 448) if rng.random() < 0.8 else 32 * _log(rng, 28, 640)   # 896 .. 28672
    k = 128 * max(7, k // 128) if rng.random() < 0.5 else k
    group = rng.choices([32, 64, 128, k], [15, 25, 40, 20] if quant == "int4" else [5, 15, 20, 60])[0]
    zeros = rng.random() < (0.6 if quant == "int4" else 0.25)
    if kind == "step":
        h = min(128 * _log(rng, 28, 224), MAX_WEIGHTS // 2 // k // 128 * 128)       # 3584 .. 28672
        k = 128 * max(7, k // 128)
        group = k if group not in (32, 64, 128) else group
        return {"kind": kind, "m": _log(rng, 1, 32), "k": min(k, 8192), "h": h, "quant": quant,
                "group": group if group <= 128 else 32768, "dtype": dtype, "zeros": zeros}
    n = min(_log(rng, 512, 57344), MAX_WEIGHTS // k)
    if rng.random() < 0.75:
        n = 64 * max(1, n // 64)
    if kind == "dequantize":
        flat = dtype == "fp16" and (n * k) % group == 0 and k % group == 0 and rng.random() < 0.5
        n = min(n, MAX_WEIGHTS // 4 // k)
        return {"kind": kind, "k": k, "n": n, "quant": quant, "group": group, "dtype": dtype,
                "zeros": zeros and not flat, "flat": flat}
    if kind == "host":
        return {"kind": kind, "m": _log(rng, 1, 64), "k": k, "n": n, "quant": quant, "group": group, "dtype": dtype,
                "zeros": zeros}
    m = min(_log(rng, 1, 4096), max(1, MAX_MACS // (n * k)))
    return {"kind": kind, "m": m, "k": k, "n": n, "quant": quant, "group": group, "dtype": dtype, "zeros": zeros,
            "epilogue": rng.choices(["none", "bias", "bias_silu", "residual"], [70, 10, 10, 10])[0]}


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _weights(gen, n, k, case):
    """Packed integers, scales and zeros of one [n, k] layer, distributed as the benchmark's are."""
    dt = DTYPES[case["dtype"]]
    g = -(-k // case["group"])
    if case["quant"] == "int4":
        wq = torch.randint(0, 256, (n, k // 2), generator=gen, device="cuda", dtype=torch.uint8)
        lo, hi = 0.005, 0.02
    else:
        wq = torch.randint(-127, 128, (n, k), generator=gen, device="cuda", dtype=torch.int8)
        lo, hi = 0.0003, 0.00125
    s = (torch.rand((n, g), generator=gen, device="cuda") * (hi - lo) + lo).to(dt)
    z = None
    if case["zeros"]:
        zp = torch.randint(0, 16, (n, g), generator=gen, device="cuda")
        z = ((zp.float() - 8.0) * s.float()).to(dt)
    return wq, s, z


def _randn(gen, shape, dtype):
    return torch.randn(shape, generator=gen, device="cuda").to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    kind, k = case["kind"], case["k"]
    st = {"case": case}
    if kind == "norm":
        st["x"], st["r"] = _randn(gen, (case["m"], k), dt), _randn(gen, (case["m"], k), dt)
        st["w"] = (1.0 + 0.1 * torch.randn(k, generator=gen, device="cuda")).to(dt)
        st["sum"] = torch.empty_like(st["x"])
        return st
    C.set_option("weights_immutable", 1)
    if kind == "step":
        m, h = case["m"], case["h"]
        x, r = _randn(gen, (m, k), dt), _randn(gen, (m, k), dt)
        nw = (1.0 + 0.1 * torch.randn(k, generator=gen, device="cuda")).to(dt)
        gu, down = _weights(gen, 2 * h, k, case), _weights(gen, k, h, case)
        y, res = torch.empty_like(x), torch.empty_like(x)
        hid, act = torch.empty_like(x), torch.empty((m, h), dtype=dt, device="cuda")
        # what the fused gate+up kernel takes whatever the layer: few tokens, groups of whole 64-byte runs
        fused = m <= 8 and case["group"] % (128 if case["quant"] == "int4" else 64) == 0
        both = None if fused else torch.empty((m, 2 * h), dtype=dt, device="cuda")

        def step():
            metal_native.fused_residual_norm(x, r, nw, out=hid, sum_out=res)
            if fused:
                metal_native.dequant_matmul_swiglu(hid, *gu, case["group"], case["quant"], out=act)
            else:
                metal_native.dequant_matmul(hid, *gu, case["group"], case["quant"], out=both)
                torch.mul(torch.nn.functional.silu(both[:, :h]), both[:, h:], out=act)
            metal_native.dequant_matmul_fused(act, *down, case["group"], case["quant"], "residual", residual=res, out=y)

        pipe = metal_native.PhasePipeline()
        pipe.auto_detect_phase(m, 1)
        st.update(replay=pipe.capture_step(step), keep=(x, r, nw, gu, down, hid, both), y=y, res=res, act=act)
        return st
    st["w"] = _weights(gen, case["n"], k, case)
    if kind == "dequantize":
        return st
    st["x"] = _randn(gen, (case["m"], k), dt)
    if kind == "host":
        st["x"] = st["x"].cpu().pin_memory()
        st["y"] = torch.empty((case["m"], case["n"]), dtype=dt, pin_memory=True)
        return st
    e = case["epilogue"]
    st["bias"] = _randn(gen, (case["n"],), dt) if e.startswith("bias") else None
    st["res"] = _randn(gen, (case["m"], case["n"]), dt) if e == "residual" else None
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        st["replay"]()
        return {"y": st["y"], "residual": st["res"], "act": st["act"]}
    if kind == "norm":
        return metal_native.fused_residual_norm(st["x"], st["r"], st["w"], sum_out=st["sum"]), st["sum"]
    if kind == "dequantize":
        wq, s, z = st["w"]
        if case["flat"]:
            return metal_native.dequantize_flat(wq.view(-1), s.view(-1), case["group"], case["quant"])
        return metal_native.dequantize(wq, s, z, case["group"], case["quant"], DTYPES[case["dtype"]])
    if kind == "host":
        metal_native.dequant_matmul(st["x"], *st["w"], case["group"], case["quant"], out=st["y"])
        metal_native.synchronize()
        return st["y"]
    if case["epilogue"] == "none":
        return metal_native.dequant_matmul(st["x"], *st["w"], case["group"], case["quant"])
    return metal_native.dequant_matmul_fused(st["x"], *st["w"], case["group"], case["quant"], case["epilogue"],
                                             bias=st["bias"], residual=st["res"])


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without, and how far a correct result may be off
# ---------------------------------------------------------------------------------------------
def _weight_bytes(n, k, case):
    g = -(-k // case["group"])
    return n * k // (2 if case["quant"] == "int4" else 1) + n * g * 2 * (2 if case["zeros"] else 1)


def work(case):
    kind, k = case["kind"], case["k"]
    if kind == "norm":
        return {"bytes": case["m"] * k * 2 * 4 + 2 * k, "flops": 0}
    if kind == "step":
        m, h = case["m"], case["h"]
        return {"bytes": _weight_bytes(2 * h, k, case) + _weight_bytes(k, h, case) + m * (4 * k + h) * 2 + 2 * k,
                "flops": 2 * m * 3 * h * k}
    n = case["n"]
    if kind == "dequantize":
        return {"bytes": _weight_bytes(n, k, case) + n * k * 2, "flops": 0}
    m = case["m"]
    extra = {"bias": n * 2, "bias_silu": n * 2, "residual": m * n * 2}.get(case.get("epilogue"), 0)
    return {"bytes": _weight_bytes(n, k, case) + m * (k + n) * 2 + extra, "flops": 2 * m * n * k}


def tolerance(case):
    """About four times the distance measured between these outputs and the same arithmetic in fp64, over the listed
    cases and a few dozen drawn ones.  What the data types give: one rounding of the result to 16 bits, for fp16
    activations above the decode sizes one rounding of each dequantised weight, and in a step the rounding of
    every intermediate tensor."""
    return TOLERANCE[case["kind"]][case["dtype"]]


TOLERANCE = {
    # measured: fp16 rel 2.9e-4, max 2.1e-3; bf16 rel 1.7e-3, max 3.9e-3
    "linear": {"fp16": {"rel": 1.2e-3, "max": 9e-3}, "bf16": {"rel": 7e-3, "max": 1.6e-2}},
    "host": {"fp16": {"rel": 1.2e-3, "max": 9e-3}, "bf16": {"rel": 7e-3, "max": 1.6e-2}},
    # measured: fp16 rel 5.8e-4, max 3.0e-3; bf16 rel 5.1e-3, max 3.7e-2
    "step": {"fp16": {"rel": 2.4e-3, "max": 1.2e-2}, "bf16": {"rel": 2e-2, "max": 0.15}},
    # measured: fp16 rel 3.1e-4, max 9.5e-4; bf16 rel 2.5e-3, max 7.7e-3
    "norm": {"fp16": {"rel": 1.2e-3, "max": 4e-3}, "bf16": {"rel": 1e-2, "max": 3e-2}},
    # the reference's own roundings, bit for bit
    "dequantize": {"fp16": "exact", "bf16": "exact"},
}


# ---------------------------------------------------------------------------------------------
# The same arithmetic in 64 bits, by torch alone
# ---------------------------------------------------------------------------------------------
def _expanded(w, k, case):
    """(q - 8) * s - z (int4; int8 without the 8) of packed rows, in fp64."""
    wq, s, z = w
    if case["quant"] == "int4":
        q = torch.empty((wq.shape[0], k), dtype=torch.float64, device=wq.device)
        q[:, 0::2], q[:, 1::2] = (wq & 15).double() - 8.0, (wq >> 4).double() - 8.0
    else:
        q = wq.double()
    g = min(case["group"], k)
    q *= s.double().repeat_interleave(g, dim=1)[:, :k]
    if z is not None:
        q -= z.double().repeat_interleave(g, dim=1)[:, :k]
    return q


def _project(x, w, case):
    """x @ W^T, expanded a block of rows at a time."""
    k = x.shape[1]
    rows = max(1, (1 << 27) // k)
    parts = [x @ _expanded([None if t is None else t[i:i + rows] for t in w], k, case).t()
             for i in range(0, w[0].shape[0], rows)]
    return torch.cat(parts, dim=1)


def _normed(x, r, w):
    s = x.double() + r.double()
    return s / torch.sqrt(s.pow(2).mean(dim=1, keepdim=True) + 1e-6) * w.double(), s


def exact(case, seed):
    """What ``run`` returns for these inputs, without any rounding between the operators."""
    kind, k = case["kind"], case["k"]
    if kind == "step":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        dt, m, h = DTYPES[case["dtype"]], case["m"], case["h"]
        x, r = _randn(gen, (m, k), dt), _randn(gen, (m, k), dt)
        nw = (1.0 + 0.1 * torch.randn(k, generator=gen, device="cuda")).to(dt)
        gu, down = _weights(gen, 2 * h, k, case), _weights(gen, k, h, case)
        hid, res = _normed(x, r, nw)
        both = _project(hid, gu, case)
        act = torch.nn.functional.silu(both[:, :h]) * both[:, h:]
        return {"y": _project(act, down, case) + res, "residual": res, "act": act}
    st = prepare(case, seed)
    if kind == "norm":
        return _normed(st["x"], st["r"], st["w"])
    if kind == "dequantize":
        w = _expanded(st["w"], k, case)
        return w.view(-1) if case["flat"] else w
    y = _project(st["x"].cuda().double(), st["w"], case)
    if kind == "host":
        return y.cpu()
    if st["bias"] is not None:
        y = y + st["bias"].double()
    if st["res"] is not None:
        y = y + st["res"].double()
    return torch.nn.functional.silu(y) if case["epilogue"] == "bias_silu" else y

"""The workloads that this framework's speed is judged by.

They are what a program that serves a block-quantised language model has the framework do on one
GPU: weights come in once and stay, activations are quantised as they arise, one to eight tokens
are decoded against streamed weights, prompts go through the tensor-core GEMM.  Layer sizes are
those of the benchmark (4096, 11008, 32000) and generic ones around them.  Weights ~ N(0, 0.02),
activations ~ N(0, 1), both quantised by the framework's own quantisers, as the benchmark does.
Everything is reached through the package's public functions; the host-buffer step goes through
the C entries of include/tcrv_emitc_host.h, which is where such a caller enters.
"""
import ctypes
import importlib
import math

import torch

tc = importlib.import_module("tianchen-rv_b200")

WEIGHT_BLOCK = {"q4_0": 18, "q8_0": 34}
SIBLING_FORMAT = {"q4_1": tc.FORMAT_Q4_1_Q8_1, "q5_0": tc.FORMAT_Q5_0_Q8_0, "q5_1": tc.FORMAT_Q5_1_Q8_1}
HEAD = 128


def listed():
    return [
        # Weights read back as fp32, for an operation that the quantised kernels do not cover.
        {"name": "dequantize_q8_0_4096x4096", "op": "dequantize", "format": "q8_0", "rows": 4096, "k": 4096},
        # The activations of a 512-token prompt on their way into the widest GEMM of a layer.
        {"name": "quantize_q8_0_512x11008", "op": "quantize", "format": "q8_0", "rows": 512, "k": 11008},
        # The output head of a decode step, one token: the largest weight stream of the step.
        {"name": "gemv_q4_0_32000x4096_b1", "op": "gemv", "weights": "q4_0", "rows": 32000, "k": 4096, "cols": 1,
         "order": "fast"},
        # The down projection for eight sequences decoded together.
        {"name": "gemv_q4_0_4096x11008_b8", "op": "gemv", "weights": "q4_0", "rows": 4096, "k": 11008, "cols": 8,
         "order": "fast"},
        # The same step on 8-bit weights: the up projection.
        {"name": "gemv_q8_0_11008x4096_b1", "op": "gemv", "weights": "q8_0", "rows": 11008, "k": 4096, "cols": 1,
         "order": "fast"},
        # A small model whose rows hold an odd number of blocks, so that no row but every eighth
        # starts on a 16-byte boundary.
        {"name": "gemv_q4_0_4000x2912_b1", "op": "gemv", "weights": "q4_0", "rows": 4000, "k": 2912, "cols": 1,
         "order": "fast"},
        # A 5-bit model's up projection, one token.
        {"name": "sibling_q5_0_11008x4096_b1", "op": "sibling", "weights": "q5_0", "rows": 11008, "k": 4096, "cols": 1},
        # One decoder layer of a decode step as a program calls it, operation by operation: norms,
        # quantisers, projections, rotation, activation and residuals (attention is the caller's).
        # Sixteen small launches: latency and the cost of a call count.
        {"name": "decode_layer_4096_11008", "op": "layer", "hidden": 4096, "ffn": 11008},
        # A decode step of a caller that keeps its activations in page-locked host memory: four
        # queued calls and one wait, in the reference's summation order (the entries' default).
        {"name": "host_step_4096_11008_32000", "op": "host_step", "hidden": 4096, "ffn": 11008, "vocab": 32000,
         "order": "strict"},
        # Prefill of a 512-token prompt against weights prepared at load time.
        {"name": "gemm_prepared_512x11008x4096", "op": "gemm", "prepared": True, "tokens": 512, "rows": 11008, "k": 4096},
        # A short prompt of no round length against the down projection.
        {"name": "gemm_prepared_77x4096x11008", "op": "gemm", "prepared": True, "tokens": 77, "rows": 4096, "k": 11008},
        # Prefill through the plain-format entry, the largest matrix: both operands are converted
        # on every call, as by a caller that has no room for a second copy of its weights.
        {"name": "gemm_plain_512x32000x4096", "op": "gemm", "prepared": False, "tokens": 512, "rows": 32000, "k": 4096},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _k(rng):
    """Elements per row: whole blocks; every second one a multiple of 256, as most models have."""
    step = rng.choice((32, 256))
    return max(512, _log(rng, 512, 11008) // step * step)


def _matrix(rng):
    """(rows, k) of a weight matrix, no more than 32000 x 4096 elements."""
    while True:
        rows, k = _log(rng, 512, 32000), _k(rng)
        if rows * k <= 32000 * 4096:
            return rows, k


def draw(rng):
    op = rng.choice(("dequantize", "quantize", "gemv", "gemv", "gemv", "sibling", "layer", "host_step", "gemm", "gemm"))
    if op == "dequantize":
        while True:
            rows, k = _log(rng, 64, 16384), _k(rng)
            if rows * k <= 64 << 20:
                return {"op": op, "format": rng.choice(("q4_0", "q8_0")), "rows": rows, "k": k}
    if op == "quantize":
        return {"op": op, "format": "q8_0", "rows": _log(rng, 1, 2048), "k": _k(rng)}
    if op == "gemv":
        rows, k = _matrix(rng)
        return {"op": op, "weights": rng.choice(("q4_0", "q4_0", "q8_0")), "rows": rows, "k": k,
                "cols": rng.choice((1, 1, 2, 3, 4, 6, 8)), "order": rng.choice(("fast", "fast", "strict"))}
    if op == "sibling":
        rows, k = _matrix(rng)
        return {"op": op, "weights": rng.choice(("q4_1", "q5_0", "q5_1")), "rows": rows, "k": k, "cols": rng.choice((1, 1, 2, 4))}
    if op == "layer":
        hidden = rng.randint(8, 40) * HEAD
        return {"op": op, "hidden": hidden, "ffn": min(13824, int(hidden * rng.uniform(2.0, 4.0)) // 32 * 32)}
    if op == "host_step":
        hidden = rng.randint(8, 32) * HEAD
        return {"op": op, "hidden": hidden, "ffn": int(hidden * rng.uniform(2.0, 2.75)) // 32 * 32,
                "vocab": _log(rng, 4000, 32000), "order": rng.choice(("strict", "fast"))}
    rows, k = _matrix(rng)
    return {"op": "gemm", "prepared": rng.random() < 0.7, "tokens": _log(rng, 9, 512), "rows": rows, "k": k}


def _normal(gen, rows, cols, std):
    return torch.randn(rows, cols, generator=gen, device="cuda", dtype=torch.float32) * std


def _weights(gen, rows, k, fmt):
    """Rows of quantised weights, made in pieces so that the fp32 form is never whole in memory."""
    quantize = tc.quantize_q4_0 if fmt == "q4_0" else tc.quantize_q8_0
    step = max(1, (64 << 20) // k)
    return torch.cat([quantize(_normal(gen, min(step, rows - r), k, 0.02)) for r in range(0, rows, step)])


def _half_bytes(t):
    return t.to(torch.float16).contiguous().view(torch.uint8)


def _sibling_weights(gen, rows, k, fmt):
    """Asymmetric 4- and 5-bit blocks (d, m, [high bits,] nibbles), symmetric 5-bit ones (d, high bits, nibbles)."""
    w = _normal(gen, rows, k, 0.02).view(rows, k // 32, 32)
    bits = 4 if fmt == "q4_1" else 5
    if fmt == "q5_0":
        d = w.abs().amax(-1, keepdim=True) / 16
        q = (w / d.clamp_min(1e-30) + 16).round().clamp(0, 31).to(torch.uint8)
        head = _half_bytes(d)
    else:
        low = w.amin(-1, keepdim=True)
        d = (w.amax(-1, keepdim=True) - low) / (2**bits - 1)
        q = ((w - low) / d.clamp_min(1e-30)).round().clamp(0, 2**bits - 1).to(torch.uint8)
        head = torch.cat([_half_bytes(d), _half_bytes(low)], -1)
    nibbles = (q[..., :16] & 15) | ((q[..., 16:] & 15) << 4)
    if bits == 4:
        return torch.cat([head, nibbles], -1).view(rows, -1)
    high = (q >> 4).view(rows, k // 32, 4, 8) << torch.arange(8, device="cuda", dtype=torch.uint8)
    return torch.cat([head, high.sum(-1, dtype=torch.uint8), nibbles], -1).view(rows, -1)


def _sibling_activations(gen, cols, k, fmt):
    x = _normal(gen, cols, k, 1.0)
    if fmt == "q5_0":
        return tc.quantize_q8_0(x)
    blocks = x.view(cols, k // 32, 32)  # Q8_1: d, d * sum(q), 32 int8
    d = blocks.abs().amax(-1, keepdim=True) / 127
    q = (blocks / d.clamp_min(1e-30)).round().to(torch.int8)
    s = d * q.sum(-1, keepdim=True, dtype=torch.float32)
    return torch.cat([_half_bytes(d), _half_bytes(s), q.view(torch.uint8)], -1).view(cols, -1)


class _HostWeights:
    """Weights in host memory, uploaded once and kept by the library as long as this object lives."""

    def __init__(self, w):
        self.host = w.cpu()
        if tc.lib().tcrv_cuda_host_register_weights(self.host.data_ptr(), self.host.numel()) != 0:
            raise RuntimeError("the weights could not be registered")

    def __del__(self):
        tc.lib().tcrv_cuda_host_unregister_weights(self.host.data_ptr())


def _host_shapes(case):
    h, f, v = case["hidden"], case["ffn"], case["vocab"]
    return [(h, h), (f, h), (h, f), (v, h)]  # (rows, k), in the order of a step


def _layer_shapes(case):
    h, f = case["hidden"], case["ffn"]
    return {"q": (h, h), "k": (h, h), "v": (h, h), "o": (h, h), "gate": (f, h), "up": (f, h), "down": (h, f)}


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op = case["op"]
    state = {"case": case}
    if op == "dequantize":
        state["w"] = _weights(gen, case["rows"], case["k"], case["format"])
    elif op == "quantize":
        state["x"] = _normal(gen, case["rows"], case["k"], 1.0)
    elif op == "gemv":
        state["w"] = _weights(gen, case["rows"], case["k"], case["weights"])
        state["x"] = tc.quantize_q8_0(_normal(gen, case["cols"], case["k"], 1.0))
        state["flags"] = tc.FLAG_STATIC_WEIGHTS | (tc.FLAG_STRICT_ORDER if case["order"] == "strict" else 0)
    elif op == "sibling":
        state["w"] = _sibling_weights(gen, case["rows"], case["k"], case["weights"])
        state["x"] = _sibling_activations(gen, case["cols"], case["k"], case["weights"])
    elif op == "gemm":
        w = _weights(gen, case["rows"], case["k"], "q4_0")
        state["w"] = tc.PreparedWeights(w) if case["prepared"] else w
        state["x"] = tc.quantize_q8_0(_normal(gen, case["tokens"], case["k"], 1.0))
    elif op == "layer":
        h, f = case["hidden"], case["ffn"]
        w = {name: _weights(gen, rows, k, "q4_0") for name, (rows, k) in _layer_shapes(case).items()}
        out = {name: torch.empty(rows, 1, device="cuda") for name, (rows, _) in _layer_shapes(case).items()}
        xq = torch.empty(1, h // 32 * 34, dtype=torch.uint8, device="cuda")
        state.update(w=w, out=out, xq=xq, x=_normal(gen, 1, h, 1.0), attention=_normal(gen, 1, h, 1.0),
                     angles=tc.rope_cache(HEAD, 17.0, 10000.0 ** (-2.0 / HEAD)),
                     qkv=tc.gemv_group_calls([(w[n], xq, out[n]) for n in ("q", "k", "v")]),
                     gate_up=tc.gemv_group_calls([(w[n], xq, out[n]) for n in ("gate", "up")]))
    else:
        state["w"] = [_HostWeights(_weights(gen, rows, k, "q4_0")) for rows, k in _host_shapes(case)]
        state["x"] = [tc.quantize_q8_0(_normal(gen, 1, k, 1.0)).cpu().pin_memory() for _, k in _host_shapes(case)]
        state["y"] = [torch.zeros(rows).pin_memory() for rows, _ in _host_shapes(case)]
        state["fold"] = 0 if case["order"] == "strict" else 1
        state["calls"] = [(ctypes.c_size_t(k), y.data_ptr(), w.host.data_ptr(), x.data_ptr(), x.numel(), rows, 1,
                           w.host.shape[1], 1)
                          for (rows, k), w, x, y in zip(_host_shapes(case), state["w"], state["x"], state["y"])]
    return state


def _run_layer(s):
    static, out, xq = tc.FLAG_STATIC_WEIGHTS, s["out"], s["xq"]
    x = s["x"]
    tc.quantize_q8_0(tc.rms_norm(x, 1e-5), out=xq)
    tc.gemv_group(s["qkv"], flags=static)
    q = tc.rope_apply(out["q"].view(-1, HEAD), s["angles"])
    k = tc.rope_apply(out["k"].view(-1, HEAD), s["angles"])
    o = tc.gemv(s["w"]["o"], tc.quantize_q8_0(s["attention"]), flags=static, out=out["o"])
    x = tc.add(x, o.view(1, -1))
    tc.quantize_q8_0(tc.rms_norm(x, 1e-5), out=xq)
    tc.gemv_group(s["gate_up"], flags=static)
    act = tc.vec_silu(out["gate"]).mul_(out["up"])
    down = tc.gemv(s["w"]["down"], tc.quantize_q8_0(act.view(1, -1)), flags=static, out=out["down"])
    return {"q": q, "k": k, "v": out["v"], "x": tc.add(x, down.view(1, -1))}


def _run_host_step(s):
    lib = tc.lib()
    lib.tcrv_cuda_host_set_fold_order(s["fold"])
    for call in s["calls"]:
        if lib.tcrv_cuda_host_gemm_q4_0_q8_0_async(*call) != 0:
            raise RuntimeError("a queued call was refused")
    if lib.tcrv_cuda_host_sync() != 0:
        raise RuntimeError("a queued call failed")
    return s["y"]


def run(state):
    op = state["case"]["op"]
    if op == "gemv":
        return tc.gemv(state["w"], state["x"], q8_weights=state["case"]["weights"] == "q8_0", flags=state["flags"])
    if op == "gemm":
        return tc.gemm(state["w"], state["x"])
    if op == "quantize":
        return tc.quantize_q8_0(state["x"])
    if op == "dequantize":
        return tc.dequantize_q4_0(state["w"]) if state["case"]["format"] == "q4_0" else tc.dequantize_q8_0(state["w"])
    if op == "sibling":
        return tc.sibling_dot_rows(SIBLING_FORMAT[state["case"]["weights"]], state["w"], state["x"])
    if op == "layer":
        return _run_layer(state)
    return _run_host_step(state)


def _gemv_work(rows, k, cols, block, act_block=34):
    blocks = k // 32
    return {"bytes": rows * blocks * block + cols * blocks * act_block + 4 * rows * cols, "flops": 2 * rows * k * cols}


def work(case):
    op = case["op"]
    if op in ("dequantize", "quantize"):
        n = case["rows"] * case["k"]
        return {"bytes": n * 4 + n // 32 * WEIGHT_BLOCK[case["format"]], "flops": 2 * n}
    if op == "gemv":
        return _gemv_work(case["rows"], case["k"], case["cols"], WEIGHT_BLOCK[case["weights"]])
    if op == "sibling":
        block, act_block = tc.SIBLING_STRIDES[SIBLING_FORMAT[case["weights"]]]
        return _gemv_work(case["rows"], case["k"], case["cols"], block, act_block)
    if op == "gemm":
        # (prepared or not: a prepared layout holds no more than the blocks do)
        return _gemv_work(case["rows"], case["k"], case["tokens"], 18)
    shapes = _layer_shapes(case).values() if op == "layer" else _host_shapes(case)
    parts = [_gemv_work(rows, k, 1, 18) for rows, k in shapes]
    return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}


def tolerance(case):
    op = case["op"]
    if op in ("dequantize", "quantize"):
        return "exact"  # one rounding per value; bytes
    if op == "layer":
        # Inside a layer fp32 sums are rounded to 8-bit activations again.  A sum that differs in its
        # last bits can move a value to the next of 255 steps: 1/127 of the block's maximum in one of
        # thousands of elements, a few 1e-4 of a row's norm for each.
        return {"rel": 1e-3, "max": 1e-2}
    return {"rel": 1e-5, "max": 1e-4}  # fp32 sums over exact integer block sums

"""Performance cases of the GEMM path: what programs built on this library call, over the sizes they call it with.

``listed()`` names the cases, ``draw(rng)`` makes further ones of the same ranges, ``prepare(case, seed)`` is what a program
holds before the call (operands on the GPU, converted weights, kernel handles and kernel arguments), ``run(state)`` is one
pass through the public entry points, ``work(case)`` the bytes and operations the path cannot do without, and
``tolerance(case)`` how far another correct implementation of the same precision may be off, and ``exact(case, seed)`` the same
results in 64 bits, by plain torch.

The kinds of call (``case["kind"]``):

* ``dispatch``  the reference's canonical flow: a kernel from a selected tile specification, kernel arguments and grid built
                once, then one blocking ``GpuRuntime.dispatch`` per call.  Latency counts: these are the small products.
* ``gemm``      ``GpuRuntime.gemm``: one bf16 product, queued, shape chosen by the caller and everything else by the library.
                Both layouts of the second operand, f32 and bf16 results, the fused epilogues.
* ``train``     one linear layer's training step on f32 tensors: ``matmul_f32`` forward, then both gradients.
* ``decode``    W4A16 products of up to sixteen rows (token generation): the projections of a layer that do not depend on
                each other, as one list, on weights converted once to the streaming layout.
* ``verify``    W4A16 products of 17 to 128 rows (batched generation, short prompts, speculative verification) on tile-major
                weights, again as a list.
* ``prefill``   W4A16 products of more than 128 rows (prompts) on the row layout.
* ``dequant``   the stand-alone INT4 dequantisation of the reference's wire format.
"""
from __future__ import annotations

import importlib
import math

import torch

t0 = importlib.import_module("rust-gpu_b200")

GROUP = 128          # quantisation group of the W4A16 weights


def listed():
    return [
        # the smallest product of the reference's own size sweep, through its blocking dispatch
        {"name": "dispatch_256", "kind": "dispatch", "m": 256, "n": 256, "k": 256},
        # a product with no convenient size: odd row count, K and N that no 16-byte rule fits, bias and ReLU
        {"name": "gemm_ragged_bias_relu", "kind": "gemm", "m": 777, "n": 1111, "k": 1357, "layout": "nt", "out": "f32", "epilogue": "bias_relu"},
        # thin decode-style product, bound by reading the weights
        {"name": "gemm_thin_128x4096x4096", "kind": "gemm", "m": 128, "n": 4096, "k": 4096, "layout": "nt", "out": "f32", "epilogue": "none"},
        # a feed-forward activation in bf16, weights as B[K,N]
        {"name": "gemm_2048_nn_silu_bf16", "kind": "gemm", "m": 2048, "n": 2048, "k": 2048, "layout": "nn", "out": "bf16", "epilogue": "silu"},
        # the headline square
        {"name": "gemm_4096", "kind": "gemm", "m": 4096, "n": 4096, "k": 4096, "layout": "nt", "out": "f32", "epilogue": "none"},
        # the largest square of the size sweep, bf16 result
        {"name": "gemm_8192_bf16", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "layout": "nt", "out": "bf16", "epilogue": "none"},
        # a linear layer of a small model: forward, gradient of the input, gradient of the weight
        {"name": "train_2048x1024x4096", "kind": "train", "m": 2048, "n": 4096, "k": 1024},
        # one token, gate and up projections of a 7B-class layer
        {"name": "decode_m1_gate_up", "kind": "decode", "m": 1, "n": 11008, "k": 4096, "count": 2},
        # sixteen sequences, four projections of the wider layer
        {"name": "decode_m16_n14336_x4", "kind": "decode", "m": 16, "n": 14336, "k": 4096, "count": 4},
        # 128 rows, gate and up projections
        {"name": "verify_m128_gate_up", "kind": "verify", "m": 128, "n": 11008, "k": 4096, "count": 2},
        # a prompt of 1024 tokens
        {"name": "prefill_m1024_n11008", "kind": "prefill", "m": 1024, "n": 11008, "k": 4096},
        # one weight matrix of the wire format to f32
        {"name": "dequant_11008x4096_f32", "kind": "dequant", "rows": 11008, "cols": 4096, "out": "f32"},
    ]


# --------------------------------------------------------------------------- further cases of the same ranges

def _log(rng, lo, hi, step=1):
    """A size between lo and hi, even over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step) * step, -(-lo // step) * step), hi // step * step))


def draw(rng):
    kind = rng.choice(["dispatch", "gemm", "gemm", "train", "decode", "decode", "verify", "prefill", "dequant"])
    if kind == "dispatch":
        step = rng.choice([1, 8, 64])
        return {"kind": kind, "m": _log(rng, 64, 1024, step), "n": _log(rng, 64, 1024, step), "k": _log(rng, 64, 2048, step)}
    if kind == "gemm":
        step = rng.choice([1, 8, 64, 128])
        # largest product: half of the listed 8192 cube, with no side longer than 8192
        m, n = _log(rng, 16, 8192, step if step == 1 else 8), _log(rng, 128, 8192, step)
        k = _log(rng, 128, 8192, step)
        return {"kind": kind, "m": m, "n": n, "k": k, "layout": rng.choice(["nt", "nt", "nn"]), "out": rng.choice(["f32", "f32", "bf16"]),
                "epilogue": rng.choice(["none", "none", "bias", "bias_relu", "silu"])}
    if kind == "train":
        step = rng.choice([8, 64])
        return {"kind": kind, "m": _log(rng, 128, 4096, step), "n": _log(rng, 128, 4096, step), "k": _log(rng, 128, 4096, step)}
    if kind == "decode":
        return {"kind": kind, "m": rng.choice([1, 1, 2, 4, 7, 8, 12, 16]), "n": _log(rng, 1024, 16384, rng.choice([8, 256])),
                "k": _log(rng, 1024, 14336, GROUP), "count": rng.choice([1, 2, 3, 4, 6])}
    if kind == "verify":
        return {"kind": kind, "m": rng.randint(17, 128), "n": _log(rng, 1024, 16384, rng.choice([8, 256])),
                "k": _log(rng, 1024, 8192, GROUP), "count": rng.choice([1, 1, 2, 3, 4])}
    if kind == "prefill":
        return {"kind": kind, "m": _log(rng, 129, 4096, rng.choice([1, 64])), "n": _log(rng, 1024, 14336, rng.choice([8, 256])),
                "k": _log(rng, 1024, 8192, GROUP)}
    return {"kind": kind, "rows": _log(rng, 256, 16384), "cols": _log(rng, 256, 16384, GROUP), "out": rng.choice(["f32", "bf16"])}


# --------------------------------------------------------------------------- inputs

_runtime = None


def _rt():
    """The process's runtime: one stream, one buffer pool, as a program keeps it."""
    global _runtime
    if _runtime is None:
        _runtime = t0.GpuRuntime(0)
    return _runtime


class _Weights:
    """Converted weights in a buffer of the runtime, given back with the state that holds them."""

    def __init__(self, buf):
        self.buf = buf
        self.addr = buf.gpu_addr()

    def __del__(self):
        self.buf.free()


def _uniform(gen, *shape):
    return (torch.rand(*shape, generator=gen, device="cuda") * 2 - 1).to(torch.bfloat16)


def _words(gen, *shape):
    return torch.randint(-2**31, 2**31, shape, generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)


def _w4(gen, n, k):
    """Row-layout INT4 weights: codes, bf16 scales in (0.001, 0.02), zero points."""
    packed = _words(gen, k // 8, n)
    scales = (torch.rand(k // GROUP, n, generator=gen, device="cuda") * 0.019 + 0.001).to(torch.bfloat16)
    zeros = _words(gen, k // GROUP, n // 8)
    return packed, scales, zeros


EPILOGUES = {"none": {}, "bias": {"epilogue": t0.EPI_BIAS_ADD_STORE_F32}, "bias_relu": {"epilogue": t0.EPI_BIAS_ADD_RELU_STORE_F32},
             "silu": {"tile_epilogue": ["silu"]}}


def _inputs(case, seed):
    """The operands of a case, made from the seed alone: what both ``prepare`` and ``exact`` start from."""
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "dequant":
        rows, cols = case["rows"], case["cols"]
        groups = rows * cols // GROUP
        return {"packed": _words(gen, rows * cols // 8), "scales": torch.rand(groups, generator=gen, device="cuda") * 0.019 + 0.001,
                "zeros": torch.randint(0, 16, (groups,), generator=gen, device="cuda", dtype=torch.int32)}
    m, n, k = case["m"], case["n"], case["k"]
    if kind in ("gemm", "dispatch"):
        nn = case.get("layout") == "nn"
        s = {"x": _uniform(gen, m, k), "b": _uniform(gen, k, n) if nn else _uniform(gen, n, k)}
        if kind == "gemm":
            s["bias"] = torch.randn(n, generator=gen, device="cuda")
        return s
    if kind == "train":
        return {"x": torch.randn(m, k, generator=gen, device="cuda"), "w": torch.randn(k, n, generator=gen, device="cuda") / math.sqrt(k),
                "dy": torch.randn(m, n, generator=gen, device="cuda")}
    problems = []
    for _ in range(case.get("count", 1)):
        w = _w4(gen, n, k)
        problems.append((w, torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)))
    return {"problems": problems}


def prepare(case, seed):
    rt, kind = _rt(), case["kind"]
    given = _inputs(case, seed)
    s = {"kind": kind, "rt": rt}
    if kind == "dequant":
        rows, cols = case["rows"], case["cols"]
        s.update(given, rows=rows, cols=cols, bf16=case["out"] == "bf16",
                 y=torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16 if case["out"] == "bf16" else torch.float32))
    elif kind in ("gemm", "dispatch"):
        m, n, k = case["m"], case["n"], case["k"]
        s.update(given, m=m, n=n, k=k, y=torch.empty(m, n, device="cuda", dtype=torch.bfloat16 if case.get("out") == "bf16" else torch.float32))
        if kind == "gemm":
            s["options"] = dict(EPILOGUES[case["epilogue"]], transpose=t0.NN if case["layout"] == "nn" else t0.NT, out_bf16=case["out"] == "bf16")
        else:
            spec = t0.tile_auto_select(m, k, n)
            s["kernel"] = rt.ensure_kernel_t0(spec)
            s["kernargs"] = t0.tile_build_kernargs_m(s["x"].data_ptr(), s["b"].data_ptr(), s["y"].data_ptr(), k, n, m, spec)
            s["grid"] = t0.tile_compute_grid(spec, m, n)
    elif kind == "train":
        m, n, k = case["m"], case["n"], case["k"]
        s.update(given, m=m, n=n, k=k)
        s.update(y=torch.empty(m, n, device="cuda"), dx=torch.empty(m, k, device="cuda"), dw=torch.empty(k, n, device="cuda"))
    else:
        m, n, k = case["m"], case["n"], case["k"]
        s.update(m=m, n=n, k=k, a=[], w=[], y=[])
        for (packed, scales, zeros), a in given["problems"]:
            s["a"].append(a)
            s["y"].append(torch.empty(m, n, device="cuda"))
            if kind == "prefill":
                s["w"].append((packed, scales, zeros))
                continue
            torch.cuda.synchronize()              # the conversion runs on the runtime's own stream
            convert = rt.w4_prepack if kind == "decode" else rt.w4_to_tiled
            s["w"].append(_Weights(convert(packed.data_ptr(), scales.data_ptr(), zeros.data_ptr(), k, n, GROUP)))
            rt.synchronize()
        if kind != "prefill":
            s["calls"] = []
            for a, w, y in zip(s["a"], s["w"], s["y"]):
                c = t0.W4A16Args()
                c.a, c.packed, c.y, c.m, c.n, c.k, c.group = a.data_ptr(), w.addr, y.data_ptr(), m, n, k, GROUP
                s["calls"].append(c)
    torch.cuda.synchronize()                      # torch's stream made the inputs, the runtime's stream reads them
    return s


# --------------------------------------------------------------------------- one pass

def run(s):
    rt, kind = s["rt"], s["kind"]
    if kind == "gemm":
        rt.gemm(s["x"].data_ptr(), s["b"].data_ptr(), s["y"].data_ptr(), s["m"], s["n"], s["k"], bias=s["bias"].data_ptr(), **s["options"])
        return s["y"]
    if kind == "dispatch":
        rt.dispatch(s["kernel"], s["grid"], s["kernargs"])
        return s["y"]
    if kind == "train":
        x, w, dy, m, n, k = s["x"].data_ptr(), s["w"].data_ptr(), s["dy"].data_ptr(), s["m"], s["n"], s["k"]
        rt.matmul_f32(x, w, s["y"].data_ptr(), m, k, n)
        rt.matmul_f32_backward_data(dy, w, s["dx"].data_ptr(), m, k, n)
        rt.matmul_f32_backward_weight(x, dy, s["dw"].data_ptr(), m, k, n)
        return [s["y"], s["dx"], s["dw"]]
    if kind == "decode":
        rt.w4a16_gemm_prepacked_batch(s["calls"])
        return s["y"]
    if kind == "verify":
        rt.w4a16_gemm_tiled_grouped(s["calls"])
        return s["y"]
    if kind == "prefill":
        packed, scales, zeros = s["w"][0]
        rt.w4a16_gemm(s["a"][0].data_ptr(), packed.data_ptr(), scales.data_ptr(), zeros.data_ptr(), s["y"][0].data_ptr(), s["m"], s["n"], s["k"], GROUP)
        return s["y"]
    rt.dequant_int4(s["packed"].data_ptr(), s["scales"].data_ptr(), s["zeros"].data_ptr(), s["y"].data_ptr(), s["rows"], s["cols"],
                    GROUP.bit_length() - 1, s["bf16"])
    return s["y"]


# --------------------------------------------------------------------------- floors and tolerances

def work(case):
    kind = case["kind"]
    if kind == "dequant":
        n = case["rows"] * case["cols"]
        return {"bytes": n // 2 + n // GROUP * 8 + n * (2 if case["out"] == "bf16" else 4), "flops": 2 * n}
    m, n, k = case["m"], case["n"], case["k"]
    if kind in ("gemm", "dispatch"):
        out = 2 if case.get("out") == "bf16" else 4
        return {"bytes": 2 * (m * k + n * k) + out * m * n + (4 * n if "bias" in case.get("epilogue", "") else 0), "flops": 2 * m * n * k}
    if kind == "train":       # x, w, dy in; y, dx, dw out
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 6 * m * n * k}
    one = k * n // 2 + k // GROUP * n * 5 // 2 + 2 * m * k + 4 * m * n
    return {"bytes": one * case.get("count", 1), "flops": 2 * m * n * k * case.get("count", 1)}


def tolerance(case):
    if case["kind"] == "dequant":
        return "exact"
    if case.get("out") == "bf16":
        # one rounding to bf16 of sums that agree to the f32 bound below: a few values fall on the other side of a tie, one unit
        # in the last place (2^-8 to 2^-7 of the value) apart.  Measured against f64 sums rounded to bf16: up to 2.1e-4
        return {"rel": 1e-3, "max": 1.6e-2}
    # f32 accumulation of exact bf16 products in another order or in other pieces of K.  The tensor cores' accumulation error
    # grows with the length of the sum: measured against f64, 1.9e-7 at K = 256 and 1e-9 K from K = 1000 on (7.5e-6 at K = 7680)
    k = max(case["m"], case["n"], case["k"]) if case["kind"] == "train" else case["k"]
    return {"rel": max(4e-6, 4e-9 * k)}


# --------------------------------------------------------------------------- the same results in 64 bits

def _nibbles(words, dim):
    """The eight codes of each 32-bit word, lowest first, in place of dimension `dim`."""
    codes = torch.stack([(words >> (4 * i)) & 15 for i in range(8)], dim + 1)
    return codes.reshape(*words.shape[:dim], words.shape[dim] * 8, *words.shape[dim + 1:])


def exact(case, seed):
    kind, given = case["kind"], _inputs(case, seed)
    if kind == "dequant":
        codes = _nibbles(given["packed"], 0).reshape(-1, GROUP)
        return ((codes - given["zeros"][:, None]).double() * given["scales"][:, None].double()).reshape(case["rows"], case["cols"])
    if kind in ("gemm", "dispatch"):
        b = given["b"].double()
        y = given["x"].double() @ (b if case.get("layout") == "nn" else b.T)
        epilogue = case.get("epilogue", "none")
        if "bias" in epilogue:
            y += given["bias"].double()
        if epilogue == "bias_relu":
            y = y.clamp_(min=0)
        return y * torch.sigmoid(y) if epilogue == "silu" else y
    if kind == "train":                           # the operands are rounded to bf16, the products are not
        x, w, dy = (given[name].to(torch.bfloat16).double() for name in ("x", "w", "dy"))
        return [x @ w, dy @ w.T, x.T @ dy]
    out = []
    for (packed, scales, zeros), a in given["problems"]:
        z = _nibbles(zeros, 1)[:, :case["n"]].repeat_interleave(GROUP, 0)
        w = ((_nibbles(packed, 0) - z).float() * scales.float().repeat_interleave(GROUP, 0)).to(torch.bfloat16)
        out.append(a.double() @ w.double())
    return out

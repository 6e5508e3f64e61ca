"""The work that users of this library have it do, as cases that can be timed and compared.

Sizes are the projections of 7B to 70B language models (4096 x 4096, 11008 x 4096, 14336 x 4096, 28672 x 8192 and its
transpose), the token counts of serving them (one sequence, a small decode batch, a speculative or chunked batch, a
prompt) and the block formats the library serves.  Weights are made on the device and uploaded once, as a model loader
does; activations are N(0, 1).  Every case goes through `GpuKernels`, the library's host interface, with one context
per process.
"""
import importlib
import math

import torch

gk = importlib.import_module("gllm-kernels_b200")

QT = gk.QuantType
TYPES = {"q4k": QT.q4k(), "q8_0": QT.q8_0(), "mxfp4": QT.mxfp4(32), "nvfp4": QT.nvfp4(), "q6k": QT.q6k(), "q5k": QT.q5k(),
         "q4_0": QT.q4_0(), "q5_0": QT.q5_0(), "q8k": QT.q8k()}
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
MAX_FLOPS = 240e9           # a drawn case costs no more than the largest listed ones: the 512-token prompt on 28672 x 8192
MAX_ELEMENTS = 28672 * 8192  # and no drawn matrix is larger than theirs

_kernels = None


def kernels():
    """The process's context: scratch and streams are shared by all its calls, as in a serving process."""
    global _kernels
    if _kernels is None:
        _kernels = gk.GpuKernels(0)
    return _kernels


# ---- the cases -------------------------------------------------------------------------------------------------
def listed():
    return [
        # one projection for one sequence, the smallest call a decode loop makes: launches and latency
        {"name": "gemv_q4k_m1", "op": "gemv", "fmt": "q4k", "n": 4096, "k": 4096, "m": 1, "host": False},
        # a decode batch of 8 on the 7B up projection, through the reference's convention: host activations in, host result out
        {"name": "gemv_q8_0_m8_host", "op": "gemv", "fmt": "q8_0", "n": 11008, "k": 4096, "m": 8, "host": True},
        # the feed-forward blocks of two 70B layers for one sequence: the decode step's bulk, bound by the weight stream
        {"name": "ffn_decode_q4k_m1", "op": "ffn_decode", "fmt": "q4k", "d": 8192, "f": 28672, "m": 1, "layers": 2},
        # FP4 weights, a decode batch of four
        {"name": "gemv_nvfp4_m4", "op": "gemv", "fmt": "nvfp4", "n": 14336, "k": 4096, "m": 4, "host": False},
        # the format GGUF files keep their down projections in, one sequence
        {"name": "gemv_q6k_m1", "op": "gemv", "fmt": "q6k", "n": 8192, "k": 28672, "m": 1, "host": False},
        # another GGUF format with a ragged batch (speculative decoding of five tokens)
        {"name": "gemv_q5k_m5", "op": "gemv", "fmt": "q5k", "n": 11008, "k": 4096, "m": 5, "host": False},
        # a 512-token prompt on the 70B gate projection, f32 in and out
        {"name": "gemm_q4k_m512", "op": "gemm", "fmt": "q4k", "n": 28672, "k": 8192, "m": 512, "dtype": "f32"},
        # a ragged mid-size batch in bf16: many sequences decoding together
        {"name": "gemm_q8_0_m33", "op": "gemm", "fmt": "q8_0", "n": 11008, "k": 4096, "m": 33, "dtype": "bf16"},
        # the gated block of a 7B layer on a 1000-token prompt, with the formats a GGUF file mixes in one block
        {"name": "ffn_prefill_q4k_q6k", "op": "ffn_prefill", "fmt": "q4k", "fmt_down": "q6k", "d": 4096, "f": 11008, "m": 1000, "dtype": "bf16"},
        # a mixture-of-experts layer: routing, gather, one grouped product, recombination
        {"name": "moe_mxfp4", "op": "moe", "fmt": "mxfp4", "experts": 8, "top_k": 2, "n": 14336, "k": 4096, "m": 512, "dtype": "bf16"},
        # a linear layer on the FP4 tensor cores: the activations are quantized and laid out on every call
        {"name": "linear_nvfp4_m2048", "op": "linear_fp4", "fmt": "nvfp4", "n": 14336, "k": 4096, "m": 2048, "dtype": "bf16"},
        # a W8A8 linear layer with bias and SiLU: quantize, integer product, epilogue
        {"name": "linear_w8a8_m2048", "op": "linear_w8a8", "n": 11008, "k": 4096, "m": 2048, "bias": True, "act": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, lo, hi):
    """Row counts: mostly the multiples of 128 that models have, some of 16, some odd (vocabularies, shards)."""
    n = _log_int(rng, lo, hi)
    step = rng.choice((128, 128, 16, 1))
    return max(lo, n // step * step)


def _depth(rng, lo, hi, step=256):
    return max(step, _log_int(rng, lo, hi) // step * step)


def _batch(rng, most):
    return 1 if rng.random() < 0.4 else rng.randint(2, most)


def draw(rng):
    op = rng.choice(("gemv", "gemv", "ffn_decode", "gemm", "gemm", "ffn_prefill", "moe", "linear_fp4", "linear_w8a8"))
    if op == "gemv":
        k = _depth(rng, 1024, 28672)
        n = _rows(rng, 1024, min(57344, MAX_ELEMENTS // k))
        return {"op": op, "fmt": rng.choice(sorted(TYPES)), "n": n, "k": k, "m": _batch(rng, 16), "host": rng.random() < 0.2}
    if op == "ffn_decode":
        d = _depth(rng, 1024, 8192)
        f = _depth(rng, 2 * d, min(4 * d, 28672))
        return {"op": op, "fmt": rng.choice(("q4k", "q8_0", "mxfp4", "nvfp4")), "d": d, "f": f, "m": _batch(rng, 16), "layers": rng.randint(1, 2)}
    if op == "gemm":
        k = _depth(rng, 1024, 28672)
        n = _rows(rng, 1024, min(57344, MAX_ELEMENTS // k))
        m = _log_int(rng, 17, max(17, min(4096, MAX_FLOPS / (2 * n * k))))
        return {"op": op, "fmt": rng.choice(("q4k", "q4k", "q8_0", "mxfp4", "nvfp4", "q6k", "q5k", "q4_0", "q5_0")), "n": n, "k": k, "m": m,
                "dtype": rng.choice(("f32", "bf16"))}
    if op == "ffn_prefill":
        d = _depth(rng, 1024, 8192)
        f = _depth(rng, 2 * d, min(4 * d, 28672))
        m = _log_int(rng, 17, max(17, min(4096, MAX_FLOPS / (6 * d * f))))
        fmt, down = rng.choice((("q4k", "q4k"), ("q4k", "q6k"), ("q8_0", "q8_0"), ("q5k", "q6k"), ("q4_0", "q4_0"), ("mxfp4", "mxfp4")))
        return {"op": op, "fmt": fmt, "fmt_down": down, "d": d, "f": f, "m": m, "dtype": rng.choice(("f32", "bf16"))}
    if op == "moe":
        experts, top_k = rng.choice((4, 8, 16, 32)), rng.choice((1, 2, 2, 4))
        k = _depth(rng, 1024, 7168)
        n = _rows(rng, 1024, min(14336, 8 * 14336 * 4096 // (experts * k)))
        m = _log_int(rng, 16, max(16, min(4096, MAX_FLOPS / (2 * n * k * top_k))))
        return {"op": op, "fmt": rng.choice(("mxfp4", "mxfp4", "nvfp4", "q4k", "q8_0")), "experts": experts, "top_k": top_k, "n": n, "k": k,
                "m": m, "dtype": rng.choice(("f32", "bf16"))}
    k = _depth(rng, 1024, 14336)
    n = _rows(rng, 1024, min(28672, MAX_ELEMENTS // k))
    m = _log_int(rng, 32, max(32, min(4096, MAX_FLOPS / (2 * n * k))))
    if op == "linear_fp4":
        return {"op": op, "fmt": rng.choice(("nvfp4", "nvfp4", "mxfp4")), "n": n, "k": k, "m": m, "dtype": rng.choice(("f32", "bf16"))}
    return {"op": op, "n": n, "k": k, "m": m, "bias": rng.random() < 0.5, "act": rng.choice((0, 0, 2, 3))}


# ---- what a program has in hand before the call -----------------------------------------------------------------
def _f16_bytes(gen, blocks, lo, hi):
    d = torch.empty(blocks, device="cuda").uniform_(lo, hi, generator=gen)
    return d.to(torch.float16).view(torch.uint8).view(blocks, 2)


def _gguf_blocks(fmt, n, k, gen):
    """Blocks of the formats the library has no encoder for: random codes and sub-block scales, and block scales that
    give weights the size of a model's (about 0.02)."""
    qt = TYPES[fmt]
    blocks = n * (k // qt.block_size())
    b = torch.randint(0, 256, (blocks, qt.block_bytes()), dtype=torch.uint8, device="cuda", generator=gen)
    if fmt == "q6k":     # 128 ql, 64 qh, 16 signed scales, d
        b[:, 208:210] = _f16_bytes(gen, blocks, 1e-5, 3e-5)
    elif fmt == "q5k":   # d, dmin, 12 packed scales, 32 qh, 128 qs
        b[:, 0:2] = _f16_bytes(gen, blocks, 4e-5, 8e-5)
        b[:, 2:4] = _f16_bytes(gen, blocks, 6e-4, 1.2e-3)
    elif fmt == "q8k":   # d f32, 256 s8, 16 s16 block sums
        b[:, 0:4] = torch.empty(blocks, device="cuda").uniform_(1e-4, 4e-4, generator=gen).view(torch.uint8).view(blocks, 4)
        b[:, 260:292] = b[:, 4:260].view(torch.int8).view(blocks, 16, 16).sum(2, dtype=torch.int16).view(torch.uint8)
    else:                # q4_0, q5_0: d first
        b[:, 0:2] = _f16_bytes(gen, blocks, 1e-3, 5e-3)
    return b.reshape(-1)


def _weight(fmt, n, k, gen):
    kk, qt = kernels(), TYPES[fmt]
    if fmt in ("q4k", "q8_0", "mxfp4", "nvfp4"):
        dense = torch.randn((n, k), device="cuda", generator=gen).mul_(0.02)
        got = kk.quantize(qt, dense)
        blocks, scales, scale = got, None, 1.0
        if fmt == "mxfp4":
            blocks, scales = got
        elif fmt == "nvfp4":
            blocks, scale = got
        return kk.upload(qt, n, k, blocks, scales, scale)
    return kk.upload(qt, n, k, _gguf_blocks(fmt, n, k, gen))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, m = case["op"], case["m"]
    s = {"case": case, "K": kernels()}
    depth = case.get("d") or case["k"]
    x = torch.randn((m, depth), device="cuda", generator=gen).to(DTYPES[case.get("dtype", "f32")] if op != "linear_fp4" else torch.float32)
    s["x"] = x
    if op == "ffn_decode":
        s["layers"] = [(_weight(case["fmt"], 2 * case["f"], case["d"], gen), _weight(case["fmt"], case["d"], case["f"], gen))
                       for _ in range(case["layers"])]
    elif op == "ffn_prefill":
        s["w"] = _weight(case["fmt"], 2 * case["f"], case["d"], gen)
        s["down"] = _weight(case["fmt_down"], case["d"], case["f"], gen)
    elif op == "moe":
        s["experts"] = [_weight(case["fmt"], case["n"], case["k"], gen) for _ in range(case["experts"])]
        s["probs"] = torch.softmax(torch.randn((m, case["experts"]), device="cuda", generator=gen), dim=1)
    elif op == "linear_w8a8":
        b = torch.randn((case["n"], case["k"]), device="cuda", generator=gen).mul_(32).round_().clamp_(-127, 127).to(torch.int8)
        s["w"] = kernels().upload_int8(b, layout_kn=False)
        s["bias"] = torch.randn(case["n"], device="cuda", generator=gen) if case["bias"] else None
    else:
        s["w"] = _weight(case["fmt"], case["n"], case["k"], gen)
    if case.get("host"):  # page-locked buffers, as a serving program keeps them
        s["x"] = torch.empty((m, depth), dtype=torch.float32, pin_memory=True).copy_(x).numpy()
        s["y"] = torch.empty((m, case["n"]), dtype=torch.float32, pin_memory=True).numpy()
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------
def run(state):
    case, k, x = state["case"], state["K"], state["x"]
    op = case["op"]
    if op == "gemv":
        return k.matmul_host(state["w"], x, out=state["y"]) if case["host"] else k.gemv(state["w"], x)
    if op == "ffn_decode":
        # each layer adds to the residual stream and the next one reads it
        for gate_up, down in state["layers"]:
            x = x + k.ffn_decode(gate_up, down, x)
        return x
    if op == "gemm":
        return k.gemm(state["w"], x, out_dtype=x.dtype)
    if op == "ffn_prefill":
        return k.ffn_prefill(state["w"], state["down"], x, out_dtype=x.dtype)
    if op == "moe":
        seq, experts, top_k = case["m"], case["experts"], case["top_k"]
        routing = k.moe_topk(state["probs"], top_k)
        offsets, perm, inv = k.moe_route(routing, seq, experts, top_k)
        rows = k.gemm_grouped(state["experts"], k.moe_gather(x, perm, top_k), offsets)
        return {"y": k.moe_weighted_sum(rows, routing, inv, seq, top_k, experts), "expert": routing[0].view(torch.int32), "weight": routing[1]}
    if op == "linear_fp4":
        qt = TYPES[case["fmt"]]
        blocks, other = k.quantize(qt, x)
        scales, scale = (None, other) if case["fmt"] == "nvfp4" else (other, 1.0)
        return k.gemm_fp4(state["w"], k.upload(qt, case["m"], case["k"], blocks, scales, scale), out_dtype=DTYPES[case["dtype"]])
    return k.w8a8_linear(state["w"], x, 1.0 / 1600, state["bias"], case["act"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _weight_bytes(fmt, n, k):
    return n * (k // TYPES[fmt].block_size()) * TYPES[fmt].block_bytes()


def work(case):
    op, m = case["op"], case["m"]
    size = 2 if case.get("dtype") == "bf16" else 4
    if op == "ffn_decode":
        d, f, layers = case["d"], case["f"], case["layers"]
        return {"bytes": layers * (_weight_bytes(case["fmt"], 2 * f, d) + _weight_bytes(case["fmt"], d, f)) + 8 * m * d,
                "flops": layers * 6 * m * d * f}
    if op == "ffn_prefill":
        d, f = case["d"], case["f"]
        return {"bytes": _weight_bytes(case["fmt"], 2 * f, d) + _weight_bytes(case["fmt_down"], d, f) + 2 * size * m * d, "flops": 6 * m * d * f}
    n, k = case["n"], case["k"]
    if op == "gemv":
        return {"bytes": _weight_bytes(case["fmt"], n, k) + 4 * m * (k + n), "flops": 2 * m * n * k}
    if op == "gemm":
        return {"bytes": _weight_bytes(case["fmt"], n, k) + size * m * (k + n), "flops": 2 * m * n * k}
    if op == "moe":
        experts, top_k = case["experts"], case["top_k"]
        return {"bytes": min(experts, m * top_k) * _weight_bytes(case["fmt"], n, k) + m * (size * k + 4 * n + 4 * experts + 8 * top_k),
                "flops": 2 * m * top_k * n * k}
    if op == "linear_fp4":
        return {"bytes": _weight_bytes(case["fmt"], n, k) + m * (4 * k + size * n), "flops": 2 * m * n * k}
    return {"bytes": n * k + 4 * m * (k + n) + (4 * n if case["bias"] else 0), "flops": 2 * m * n * k}


# Relative 2-norm error against the same product evaluated in 64 bits on the decoded weights, times four.
#   decode: f32 activations carried as fixed point (two s8 digits per 256 elements, or s16 per 32): 2.0e-5 to 2.7e-5;
#           FP4 weights (eight E2M1 digits): 3.3e-6; a chain of two gated blocks: up to 1.2e-4
#   prefill, f32 results: operands staged in fp16, so the weight's own rounding to fp16: 7.0e-4 where a min is subtracted
#           (Q4_K, Q5_K), 2.1e-4 to 3.6e-4 otherwise; bf16 results: 1.7e-3, the rounding of the result
#   gated block, prompt: the intermediate is kept in bf16: 3.2e-3
#   FP4 x FP4 and W8A8: products exact, f32 sums or the f32 epilogue only
def tolerance(case):
    op, fmt, bf16 = case["op"], case.get("fmt"), case.get("dtype") == "bf16"
    fp4 = fmt in ("mxfp4", "nvfp4")
    if op == "gemv":
        return {"rel": 1.3e-5 if fp4 else 1e-4}
    if op == "ffn_decode":
        return {"rel": 5e-4}
    if op == "ffn_prefill":
        return {"rel": 1.3e-2}
    if op == "linear_fp4":
        return {"rel": 7e-3 if bf16 else 1e-5}
    if op == "linear_w8a8":
        return {"rel": 1e-6}
    if op == "gemm" and bf16:
        return {"rel": 7e-3}
    return {"rel": 2.8e-3 if fmt in ("q4k", "q5k") else 1.4e-3}

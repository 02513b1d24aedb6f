"""Performance cases: the calls a host program makes on the quantized-matmul path, over the sizes it makes them at.

Four kinds of case, each through the package's public entry points:

  gemv     one projection of one decode step: QwenGemvKernel.execute (one row) or execute_warp_batch (2..64 rows), called
           eagerly; Q4_K / Q5_K / Q6_K / Q8_0 weights, f32 or bf16 rows, f32 outputs.
  gemm     one projection of a prompt chunk: gemm(), bf16 rows, f32 or bf16 outputs.
  decode   one token for every sequence of a batch: a captured CudaDenseDecode step, replayed.  It covers the operators
           between the projections: embedding, norms, rope, cache append, attention, gating, residuals, argmax.
  prefill  a prompt through CudaDenseDecode.prefill in its default chunks.

Sizes are those of the repository's benchmark and tests, of the Qwen3-8B and Qwen3-32B geometries that
engine_b200.decode names, or generic.
"""
import math

import torch

import engine_b200
from engine_b200 import decode, synth

Q8_0, Q4_K, Q5_K, Q6_K = 8, 12, 13, 14
TYPES = {"q8_0": Q8_0, "q4_k": Q4_K, "q5_k": Q5_K, "q6_k": Q6_K}

# The generators of engine_b200.synth make weights of magnitude three; a trained network's projections of a normalised row
# are of order one.  The norm vectors in front of the projections carry the difference.
NORM_SCALE = 1.0 / 256.0

_stream = None


def _gemv(name, quant, members, n, k, dtype):
    return {"name": name, "kind": "gemv", "quant": quant, "members": members, "n": n, "k": k, "dtype": dtype}


def _gemm(name, quant, tokens, n, k, out):
    return {"name": name, "kind": "gemm", "quant": quant, "tokens": tokens, "n": n, "k": k, "out": out}


def _decode(name, members, context, layers, vocabulary):
    return {"name": name, "kind": "decode", "members": members, "context": context, "layers": layers, "vocabulary": vocabulary}


def listed():
    return [
        # the smallest projection of a step: attn_v of the 8B geometry for one sequence, a few megabytes
        _gemv("gemv_q6k_m1_1024x4096", "q6_k", 1, 1024, 4096, "f32"),
        # one sequence's gate or up projection
        _gemv("gemv_q4k_m1_12288x4096", "q4_k", 1, 12288, 4096, "f32"),
        # a model file kept in 8-bit blocks
        _gemv("gemv_q8_0_m1_4096x4096", "q8_0", 1, 4096, 4096, "f32"),
        # a few sequences together, the 32B geometry's attn_v: Q6_K rows of 20 blocks, which do not start on 16-byte boundaries
        _gemv("gemv_q6k_m3_1024x5120", "q6_k", 3, 1024, 5120, "bf16"),
        # an ordinary decode batch
        _gemv("gemv_q4k_m16_12288x4096", "q4_k", 16, 12288, 4096, "bf16"),
        # the largest decode batch, the down projection
        _gemv("gemv_q6k_m64_4096x12288", "q6_k", 64, 4096, 12288, "bf16"),
        # the last, ragged chunk of a prompt
        _gemm("gemm_q5k_t173_5120x5120", "q5_k", 173, 5120, 5120, "bf16"),
        # a full chunk of a prompt through the gate or up projection
        _gemm("gemm_q4k_t512_12288x4096", "q4_k", 512, 12288, 4096, "f32"),
        # a long prompt in one call through the down projection
        _gemm("gemm_q6k_t2048_4096x12288", "q6_k", 2048, 4096, 12288, "f32"),
        # the whole 8B geometry for one sequence in the middle of its answer
        _decode("decode_b1_ctx2048", 1, 2048, 36, 151936),
        # a serving batch: a stack of 8B layers with a vocabulary in proportion
        _decode("decode_b32_ctx2048", 32, 2048, 8, 32768),
        # a prompt of odd length: three full chunks and a ragged one
        {"name": "prefill_t1987", "kind": "prefill", "tokens": 1987, "layers": 4, "vocabulary": 32768},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(("gemv", "gemm", "decode", "prefill"), weights=(6, 3, 2, 1))[0]
    quant = rng.choice(sorted(TYPES))
    if kind == "gemv":
        members = rng.choice((1, 1, _log_int(rng, 2, 8), _log_int(rng, 9, 64)))
        k = 256 * _log_int(rng, 4, 48)
        if quant == "q8_0" and members <= 8 and rng.random() < 0.5:
            k -= 32 * rng.randrange(8)        # blocks of 32: the only format whose rows need not be whole super-blocks
        n = _log_int(rng, 256, 16384)
        n = n if rng.random() < 0.5 else (n + 63) // 64 * 64
        # a decode step keeps its rows in f32; a host that batches more than eight brings bf16
        dtype = "bf16" if members > 8 else rng.choice(("f32", "bf16"))
        return {"kind": kind, "quant": quant, "members": members, "n": n, "k": k, "dtype": dtype}
    if kind == "gemm":
        n = _log_int(rng, 512, 16384)
        n = n if rng.random() < 0.5 else (n + 63) // 64 * 64
        return {"kind": kind, "quant": quant, "tokens": _log_int(rng, 65, 2048), "n": n, "k": 256 * _log_int(rng, 4, 48),
                "out": rng.choice(("f32", "bf16"))}
    if kind == "decode":
        members = _log_int(rng, 1, 64)
        return {"kind": kind, "members": members, "context": _log_int(rng, 60, min(4096, 65536 // members)), "layers": rng.randint(3, 8),
                "vocabulary": rng.choice((8192, 32000, 32768))}
    return {"kind": kind, "tokens": _log_int(rng, 65, 1900), "layers": rng.randint(2, 4), "vocabulary": 32768}


def _geometry(case):
    base = decode.DenseGeometry.qwen3_8b(case["layers"])
    return decode.DenseGeometry(base.hidden, base.layers, base.q_heads, base.kv_heads, base.head_dim, base.intermediate, case["vocabulary"])


def _serving_stream(device):
    """The stream a serving program enqueues its steps on: each step waits for the one before it, whichever sequences they hold."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream(device)
    return _stream


def _model(case, seed, members, max_context):
    """A random-init decoder, as a serving program keeps one."""
    device = torch.device("cuda", 0)
    context = engine_b200.RibnContext(device, _serving_stream(device))
    geometry = _geometry(case)
    with torch.cuda.stream(context.stream):
        weights = decode.random_weights(context, geometry, seed=seed)
        for name, vector in weights.vectors.items():
            if name.endswith(("attn_norm", "ffn_norm", "output_norm")):
                vector.mul_(NORM_SCALE)
        decoder = decode.CudaDenseDecode(context, geometry, weights, members, max_context)
    return decoder


def prepare(case, seed):
    device = torch.device("cuda", 0)
    generator = torch.Generator(device=device)
    generator.manual_seed(seed)
    if case["kind"] == "decode":
        decoder = _model(case, seed, case["members"], case["context"] + 8)
        decoder.fill_context(case["context"], seed=seed)
        decoder.capture()
        torch.cuda.synchronize()
        return {"kind": "decode", "decoder": decoder, "position": case["context"]}
    if case["kind"] == "prefill":
        decoder = _model(case, seed, 1, case["tokens"] + 8)
        prompt = torch.randint(0, case["vocabulary"], (case["tokens"],), device=device, generator=generator, dtype=torch.int32)
        torch.cuda.synchronize()
        return {"kind": "prefill", "decoder": decoder, "prompt": prompt}
    context = engine_b200.RibnContext(device)
    value_type = TYPES[case["quant"]]
    data = synth.random_weight_device(value_type, case["k"], case["n"], seed=seed, device=device)
    weight = engine_b200.CudaQuantizedWeight(engine_b200.WeightTensorSpec.new("weight", [case["k"], case["n"]]), value_type, data)
    rows = case["members"] if case["kind"] == "gemv" else case["tokens"]
    x = torch.randn(rows, case["k"], device=device, generator=generator)
    if case["kind"] == "gemm":
        y = torch.empty(rows, case["n"], device=device, dtype=torch.float32 if case["out"] == "f32" else torch.bfloat16)
        return {"kind": "gemm", "context": context, "weight": weight, "x": x.to(torch.bfloat16), "y": y}
    kernel = engine_b200.QwenGemvKernel.from_value_type(value_type, context)
    return {"kind": "gemv", "kernel": kernel, "weight": weight, "x": x if case["dtype"] == "f32" else x.to(torch.bfloat16), "members": rows,
            "y": torch.empty(rows, case["n"], device=device)}


def run(state):
    kind = state["kind"]
    if kind == "gemv":
        if state["members"] == 1:
            state["kernel"].execute(state["weight"], state["x"], state["y"])
        else:
            state["kernel"].execute_warp_batch(state["weight"], state["x"], state["y"], state["members"])
        return state["y"]
    if kind == "gemm":
        engine_b200.gemm(state["context"], state["weight"], state["x"], state["y"])
        return state["y"]
    decoder = state["decoder"]
    if kind == "decode":
        # without `advance` a replay leaves tokens and positions alone, so that a step can be repeated: it writes its cache slot again
        decoder.replay()
        at = state["position"]
        return {"logits": decoder.logits, "keys": decoder.k_cache[:, :, :, at], "values": decoder.v_cache[:, :, :, at]}
    count = state["prompt"].numel()
    decoder.prefill(state["prompt"])
    return {"logits": decoder.logits, "keys": decoder.k_cache[:, 0, :, :count], "values": decoder.v_cache[:, 0, :, :count]}


def _stack(case):
    """(weights of the layers, encoded bytes of the layers, weights of the head, encoded bytes of the head)"""
    g = _geometry(case)
    q, kv = g.q_heads * g.head_dim, g.kv_heads * g.head_dim
    shapes = [("attn_q", g.hidden, q), ("attn_k", g.hidden, kv), ("attn_v", g.hidden, kv), ("attn_output", q, g.hidden),
              ("ffn_gate", g.hidden, g.intermediate), ("ffn_up", g.hidden, g.intermediate), ("ffn_down", g.intermediate, g.hidden)]
    count = sum(k * n for _, k, n in shapes) * g.layers
    size = sum(synth.encoded_bytes(decode.VALUE_TYPES[kind], k, n) for kind, k, n in shapes) * g.layers
    return count, size, g.hidden * g.vocabulary, synth.encoded_bytes(decode.VALUE_TYPES["output"], g.hidden, g.vocabulary)


def work(case):
    """Bytes: encoded weights, inputs and outputs once.  Operations: the products, and those of the attention."""
    if case["kind"] in ("gemv", "gemm"):
        k, n = case["k"], case["n"]
        rows = case["members"] if case["kind"] == "gemv" else case["tokens"]
        x_size = 4 if case.get("dtype") == "f32" else 2
        y_size = 2 if case.get("out") == "bf16" else 4
        return {"bytes": synth.encoded_bytes(TYPES[case["quant"]], k, n) + rows * (k * x_size + n * y_size), "flops": 2 * rows * k * n}
    g = _geometry(case)
    count, size, head_count, head_size = _stack(case)
    kv_token = g.layers * g.kv_heads * g.head_dim * 2 * 2          # f16 keys and values of one token
    if case["kind"] == "decode":
        m, context = case["members"], case["context"] + 1
        return {"bytes": size + head_size + m * context * kv_token + m * g.vocabulary * 4,
                "flops": 2 * m * (count + head_count) + 4 * m * context * g.layers * g.q_heads * g.head_dim}
    t = case["tokens"]
    return {"bytes": size + head_size + t * kv_token + g.vocabulary * 4,
            "flops": 2 * (t * count + head_count) + 2 * t * (t + 1) * g.layers * g.q_heads * g.head_dim}


def tolerance(case):
    if case["kind"] == "gemv":
        # up to eight rows keep the weights exact and the rows to 16 bits or more; wider batches multiply in f16
        return {"rel": 1e-4} if case["members"] <= 8 else {"rel": 1e-3}
    if case["kind"] == "gemm":
        return {"rel": 5e-3} if case["out"] == "bf16" else {"rel": 1e-3}     # f16 products; a bf16 output is rounded once more
    if case["kind"] == "decode":
        # up to eight sequences: f32 rows, an f16 cache; wider batches multiply in f16 in every projection
        return {"rel": 2e-3} if case["members"] <= 8 else {"rel": 1e-2}
    return {"rel": 1e-2}                                                         # bf16 rows between the operators

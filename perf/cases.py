"""The work that is timed when this library's speed is looked at: what a program that serves
GGUF, NVFP4 and FP8 models has it do, through the operators of `layerstormgemmkernels_b200.ops`.

Families (`case["op"]`):
  gemv     one projection of one decode step, an eager operator call: latency and host cost count
  decode   the seven projections of a decoder layer at 1 to 8 rows, replayed from a CUDA graph as
           a decode loop runs them; activations in device or in page-locked host memory
  linear   a projection of a prompt chunk or of a batch of sequences on the tensor cores
  moe      a whole MoE layer (route, sort, expert block, combine); decode-sized token counts are
           replayed from a CUDA graph, prompt-sized ones are called eagerly
  nvfp4_experts, nvfp4_linear, fp8_linear   the same with NVFP4 and FP8 weights, the activation
           quantizers included
Weights are N(0, 0.02) in the packed format of the type, activations N(0, 1).
"""
import math

import torch

from layerstormgemmkernels_b200 import ops
from layerstormgemmkernels_b200.formats import BLOCK_BYTES, BLOCK_VALUES, GGUF_TYPES

# (projection, N, K, which of the layer's activations it reads)
LAYER = (("q", 4096, 4096, 0), ("k", 1024, 4096, 0), ("v", 1024, 4096, 0), ("o", 4096, 4096, 1),
         ("gate", 14336, 4096, 2), ("up", 14336, 4096, 2), ("down", 4096, 14336, 3))
GRAPH_TOKENS = 256      # MoE layers of up to this many tokens are decode steps: replayed from a graph


def listed():
    return [
        # smallest call: one 4096 x 4096 projection for one token
        {"name": "gemv_q4_0_m1", "op": "gemv", "type": "Q4_0", "M": 1, "N": 4096, "K": 4096},
        # single-stream decoding, activations and results in host memory
        {"name": "decode_q4_k_m1_host", "op": "decode", "type": "Q4_K", "M": 1, "host": True},
        # batched decoding of eight sequences with the six-bit type
        {"name": "decode_q6_k_m8", "op": "decode", "type": "Q6_K", "M": 8, "host": False},
        # a batch of sequences or of speculated tokens, too many for the mat-vec kernels
        {"name": "linear_q4_k_m48", "op": "linear", "type": "Q4_K", "M": 48, "N": 14336, "K": 4096},
        # prefill: a full chunk, and a ragged one with the six-bit type and the long K of a down projection
        {"name": "linear_q4_k_m4096", "op": "linear", "type": "Q4_K", "M": 4096, "N": 14336, "K": 4096},
        {"name": "linear_q6_k_m1000", "op": "linear", "type": "Q6_K", "M": 1000, "N": 4096, "K": 14336},
        # MoE layer (128 experts, top-8): one sequence, a decode batch, a prompt chunk
        {"name": "moe_q4_k_t1", "op": "moe", "type": "Q4_K", "T": 1, "E": 128, "top_k": 8, "H": 2048, "I": 768},
        {"name": "moe_q4_k_t64", "op": "moe", "type": "Q4_K", "T": 64, "E": 128, "top_k": 8, "H": 2048, "I": 768},
        {"name": "moe_q4_k_t4096", "op": "moe", "type": "Q4_K", "T": 4096, "E": 128, "top_k": 8, "H": 2048, "I": 768},
        # NVFP4 expert block (8 experts, top-2) over a prompt chunk, rows grouped by expert
        {"name": "nvfp4_experts_t4096", "op": "nvfp4_experts", "T": 4096, "E": 8, "top_k": 2, "H": 4096, "I": 14336},
        # NVFP4 projection of a decode batch with a ragged row count
        {"name": "nvfp4_linear_m77", "op": "nvfp4_linear", "M": 77, "N": 4096, "K": 14336},
        # FP8 projection of a prompt chunk, activations quantized on the way
        {"name": "fp8_linear_m2048", "op": "fp8_linear", "M": 2048, "N": 4096, "K": 4096},
    ]


def _log(rng, lo, hi):
    """Spread over the logarithm of lo..hi, odd numbers among them."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["gemv", "decode", "linear", "linear", "moe", "moe", "nvfp4_experts", "nvfp4_linear", "fp8_linear"])
    types = ["Q4_K", "Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0"]
    if op == "gemv":
        t = rng.choice(types)
        return {"op": op, "type": t, "M": rng.randint(1, 8), "N": _log(rng, 1024, 16384), "K": 256 * _log(rng, 4, 56)}
    if op == "decode":
        return {"op": op, "type": rng.choice(types), "M": rng.randint(1, 8), "host": rng.random() < 0.5}
    if op == "linear":
        return {"op": op, "type": rng.choice(types), "M": _log(rng, 9, 4096), "N": _log(rng, 1024, 14336),
                "K": 256 * _log(rng, 4, 56)}
    if op == "moe":
        # decode steps and prompts, few wide or many narrow experts
        E, k, H, I = rng.choice([(128, 8, 2048, 768), (64, 6, 2048, 1024), (32, 4, 2048, 1536)])
        return {"op": op, "type": rng.choice(["Q4_K", "Q4_K", "Q6_K"]), "T": _log(rng, 1, 4096), "E": E, "top_k": k,
                "H": H, "I": I}
    if op == "nvfp4_experts":
        return {"op": op, "T": _log(rng, 16, 4096), "E": 8, "top_k": 2, "H": rng.choice([2048, 4096]),
                "I": rng.choice([4096, 7168, 14336])}
    if op == "nvfp4_linear":
        return {"op": op, "M": _log(rng, 1, 4096), "N": 32 * _log(rng, 32, 448), "K": 64 * _log(rng, 16, 224)}
    return {"op": op, "M": _log(rng, 1, 4096), "N": 8 * _log(rng, 128, 1792), "K": 128 * _log(rng, 8, 112)}


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
def _randn(gen, *shape, std=1.0, dtype=torch.float32):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, std, generator=gen).to(dtype)


def _f16_bytes(x):
    return x.to(torch.float16).unsqueeze(-1).view(torch.uint8)


def _k4_scale_bytes(sc, mn):
    """Eight 6-bit scales and minima of a super-block -> the 12-byte field of Q4_K and Q5_K."""
    return torch.cat([sc[..., :4] | ((sc[..., 4:] >> 4) << 6), mn[..., :4] | ((mn[..., 4:] >> 4) << 6),
                      (sc[..., 4:] & 15) | ((mn[..., 4:] & 15) << 4)], -1)


def _pack(w, type_name):
    """float [rows, K] on the GPU -> packed blocks uint8 [rows, bytes]."""
    rows, K = w.shape
    if type_name in ("Q4_K", "Q5_K"):
        top = 15 if type_name == "Q4_K" else 31
        b = w.view(rows, K // 256, 8, 32)
        mn = (-b.amin(-1)).clamp_min(0)
        sc = (b.amax(-1) + mn) / top
        d, dmin = (sc.amax(-1) / 63).half().float(), (mn.amax(-1) / 63).half().float()
        scq = (sc / d.unsqueeze(-1)).round().clamp(0, 63)
        mnq = (mn / dmin.unsqueeze(-1)).round().clamp(0, 63)
        q = (b + (dmin.unsqueeze(-1) * mnq).unsqueeze(-1)) / (d.unsqueeze(-1) * scq).unsqueeze(-1)
        q = q.nan_to_num(0.0, 0.0, 0.0).round().clamp(0, top).to(torch.uint8)
        parts = [_f16_bytes(d), _f16_bytes(dmin), _k4_scale_bytes(scq.to(torch.uint8), mnq.to(torch.uint8))]
        if type_name == "Q5_K":
            parts.append(sum((q[:, :, j] >> 4) << j for j in range(8)))
        low = q & 15
        parts.append((low[:, :, 0::2] | (low[:, :, 1::2] << 4)).flatten(-2))
        out = torch.cat(parts, -1)
    elif type_name == "Q6_K":
        b = w.view(rows, K // 256, 16, 16)
        s = b.abs().amax(-1) / 32
        d = (s.amax(-1) / 127).half().float()
        sc = (s / d.unsqueeze(-1)).round().clamp(0, 127)
        q = (b / (d.unsqueeze(-1) * sc).unsqueeze(-1)).nan_to_num(0.0, 0.0, 0.0).round().clamp(-32, 31) + 32
        q = q.to(torch.uint8).view(rows, K // 256, 2, 4, 32)
        low, high = q & 15, q >> 4
        ql = torch.cat([low[:, :, :, 0] | (low[:, :, :, 2] << 4), low[:, :, :, 1] | (low[:, :, :, 3] << 4)], -1)
        qh = high[:, :, :, 0] | (high[:, :, :, 1] << 2) | (high[:, :, :, 2] << 4) | (high[:, :, :, 3] << 6)
        out = torch.cat([ql.flatten(-2), qh.flatten(-2), sc.to(torch.uint8), _f16_bytes(d)], -1)
    elif type_name == "Q8_0":
        b = w.view(rows, K // 32, 32)
        d = (b.abs().amax(-1) / 127).half().float()
        q = (b / d.unsqueeze(-1)).round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
        out = torch.cat([_f16_bytes(d), q], -1)
    else:   # Q4_0
        b = w.view(rows, K // 32, 32)
        d = (b.gather(-1, b.abs().argmax(-1, keepdim=True)) / -8).half().float()
        q = ((b / d).nan_to_num(0.0, 0.0, 0.0).round() + 8).clamp(0, 15).to(torch.uint8)
        out = torch.cat([_f16_bytes(d.squeeze(-1)), q[..., :16] | (q[..., 16:] << 4)], -1)
    return out.reshape(rows, -1).contiguous()


def _weight(gen, type_name, rows, K):
    """Packed N(0, 0.02) weights, made in pieces of at most 64 M values."""
    piece = max(1, (1 << 26) // K)
    return torch.cat([_pack(_randn(gen, min(piece, rows - r), K, std=0.02), type_name) for r in range(0, rows, piece)])


def _experts(gen, type_name, E, N, K):
    """E packed matrices and the device array of their addresses."""
    w = _weight(gen, type_name, E * N, K).view(E, N, -1)
    return w, torch.tensor([w[e].data_ptr() for e in range(E)], dtype=torch.int64, device="cuda")


def _nvfp4_weight(gen, N, K):
    """N(0, 0.02) weight -> (codes, interleaved scales, tensor scale)."""
    w = _randn(gen, N, K, std=0.02)
    s = float(w.abs().amax()) / 6.0
    codes, scales = ops.bf16_to_nvfp4((w / s).to(torch.bfloat16))
    return codes, scales, s


def _captured(call):
    """The call recorded into a CUDA graph; returns (graph, its outputs)."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return graph, out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)
    s = dict(case)
    op = case["op"]
    if "type" in case:
        s["t"] = GGUF_TYPES[case["type"]]
    if op in ("gemv", "linear"):
        s["x"] = _randn(gen, case["M"], case["K"], dtype=torch.bfloat16)
        s["w"] = _weight(gen, case["type"], case["N"], case["K"])
    elif op == "decode":
        M = case["M"]
        s["w"] = [_weight(gen, case["type"], n, k) for _, n, k, _ in LAYER]
        s["x"] = [_randn(gen, M, k, dtype=torch.bfloat16) for k in (4096, 4096, 4096, 14336)]
        if case["host"]:
            s["x"] = [x.cpu().pin_memory() for x in s["x"]]
            s["batch"] = ops.HostMmvqBatch([(s["x"][a], w, s["t"], n, k, None)
                                            for w, (_, n, k, a) in zip(s["w"], LAYER)]).capture()
        else:
            s["graph"], s["out"] = _captured(lambda: _decode_layer(s))
    elif op == "moe":
        E, H, I = case["E"], case["H"], case["I"]
        s["gate"], s["gate_p"] = _experts(gen, case["type"], E, I, H)
        s["up"], s["up_p"] = _experts(gen, case["type"], E, I, H)
        s["down"], s["down_p"] = _experts(gen, case["type"], E, H, I)
        s["x"] = _randn(gen, case["T"], H, dtype=torch.bfloat16)
        s["logits"] = _randn(gen, case["T"], E)
        if case["T"] <= GRAPH_TOKENS:
            s["graph"], s["out"] = _captured(lambda: _moe_layer(s))
    elif op == "nvfp4_experts":
        E, H, I = case["E"], case["H"], case["I"]
        for name, n, k in (("gate", I, H), ("up", I, H), ("down", H, I)):
            parts = [_nvfp4_weight(gen, n, k) for _ in range(E)]
            s[name] = (torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts]),
                       torch.tensor([p[2] for p in parts], dtype=torch.float32, device="cuda"))
        rows = case["T"] * case["top_k"]
        idx, _ = ops.moe_route(_randn(gen, case["T"], E), case["top_k"])
        s["offs"] = ops.moe_permutation(idx, E)[0]
        s["x"] = _randn(gen, rows, H, dtype=torch.bfloat16)
        m = (s["offs"][1:] - s["offs"][:-1]).tolist()
        s["sizes_i"] = torch.tensor([[r, I, H] for r in m], dtype=torch.int32, device="cuda")
        s["sizes_h"] = torch.tensor([[r, H, I] for r in m], dtype=torch.int32, device="cuda")
        s["g"], s["u"] = (torch.empty((rows, I), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        s["y"] = torch.empty((rows, H), dtype=torch.bfloat16, device="cuda")
    elif op == "nvfp4_linear":
        s["x"] = _randn(gen, case["M"], case["K"], dtype=torch.bfloat16)
        s["w"], s["ws"], s["s2"] = _nvfp4_weight(gen, case["N"], case["K"])
    else:
        s["x"] = _randn(gen, case["M"], case["K"], dtype=torch.bfloat16)
        s["w"], s["ws"] = ops.weight_fp8_quant(_randn(gen, case["N"], case["K"], std=0.02, dtype=torch.bfloat16))
    return s


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def _decode_layer(s):
    w, x, t = s["w"], s["x"], s["t"]
    out = []
    for a in range(4):
        out += ops.gguf_mmvq_batch(x[a], [(w[i], n) for i, (_, n, _, b) in enumerate(LAYER) if b == a], t)
    return out


def _moe_layer(s):
    H, I, k = s["H"], s["I"], s["top_k"]
    idx, weights = ops.moe_route(s["logits"], k)
    offs, perm, inv = ops.moe_permutation(idx, s["E"])
    experts = (offs, s["gate_p"], s["up_p"], s["down_p"], s["t"], H, I)
    if s["type"] == "Q4_K":
        y = ops.gguf_moe_ffn(s["x"], *experts, perm=perm, top_k=k)
    else:   # prompt-sized batches of the other types take rows that the caller has gathered
        y = ops.gguf_moe_ffn(ops.moe_permute(s["x"], perm, k), *experts)
    return ops.moe_unpermute(y, inv, weights)


def run(s):
    op = s["op"]
    if "graph" in s:
        s["graph"].replay()
        return s["out"]
    if op == "gemv":
        return ops.gguf_mmvq(s["x"], s["w"], s["t"], s["N"], s["K"])
    if op == "decode":
        return s["batch"].run()
    if op == "linear":
        return ops.gguf_mmq(s["x"], s["w"], s["t"], s["N"], s["K"])
    if op == "moe":
        return _moe_layer(s)
    if op == "nvfp4_experts":
        offs, H, I = s["offs"], s["H"], s["I"]
        q, qs, sfo = ops.bf16_to_nvfp4_grouped(s["x"], offs)
        for name, out in (("gate", s["g"]), ("up", s["u"])):
            w, ws, alpha = s[name]
            ops.nvfp4_grouped_gemm(q, w, out, qs, ws, alpha, offs, sfo, s["sizes_i"], I, H, "bf16")
        q, qs, sfo = ops.silu_mul_to_nvfp4_grouped(s["g"], s["u"], offs)
        w, ws, alpha = s["down"]
        return ops.nvfp4_grouped_gemm(q, w, s["y"], qs, ws, alpha, offs, sfo, s["sizes_h"], H, I, "bf16")
    if op == "nvfp4_linear":
        return ops.nvfp4_gemm_from_bf16(s["x"], s["w"], s["ws"], s["s2"])
    q, qs = ops.dynamic_fp8_quant(s["x"], m_major_scales=True)
    return ops.fp8_gemm(q, s["w"], qs, s["ws"], s["M"], s["N"], s["K"], "bf16")


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    op = case["op"]
    packed = BLOCK_BYTES[GGUF_TYPES[case["type"]]] / BLOCK_VALUES[GGUF_TYPES[case["type"]]] if "type" in case else 0
    if op == "decode":
        values = sum(n * k for _, n, k, _ in LAYER)
        ends = case["M"] * 2 * (3 * 4096 + 14336 + sum(n for _, n, _, _ in LAYER))
        return {"bytes": values * packed + ends, "flops": 2 * case["M"] * values}
    if op in ("moe", "nvfp4_experts"):
        T, E, k, H, I = (case[n] for n in ("T", "E", "top_k", "H", "I"))
        hit = E * (1 - (1 - k / E) ** T)      # experts that some token is routed to
        per_value = packed if op == "moe" else 0.5 + 1 / 16
        ends = 2 * T * H * 2 + T * E * 4 if op == "moe" else 2 * T * k * H * 2
        return {"bytes": hit * 3 * H * I * per_value + ends, "flops": 6 * T * k * H * I}
    M, N, K = case["M"], case["N"], case["K"]
    per_value = packed or (0.5 + 1 / 16 if op == "nvfp4_linear" else 1 + 4 / 128 / 128)
    return {"bytes": N * K * per_value + 2 * M * (N + K), "flops": 2 * M * N * K}


def tolerance(case):
    """About four times what the path differs by from the same path with its sums in 64 bits.

    bf16 results alone differ by 1.7e-3 (largest: 4e-3 of the value); fp16 operands on the tensor
    cores make that 1.8e-3 (6e-3, a result next to a rounding limit 8e-3).  In a prompt-sized MoE layer
    they also move gate and up by a bf16 place now and then, and with it the 8-bit code of an
    activation: 5.9e-3 (4e-2)."""
    if case["op"] == "moe" and case["T"] * case["top_k"] // case["E"] > 8:
        return {"rel": 2.4e-2, "max": 0.16}
    return {"rel": 7e-3, "max": 0.032}

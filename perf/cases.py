"""The calls that a program built on this library spends its time in, as cases that can be timed and compared.

Four kinds, all through the public entry points:
  fc         one packed-weight Linear (capi.Weight.matmul) on device tensors: the decode shapes (1 to 16 rows, bound by the
             stream of weights) and the prefill shapes (17 rows and more), with bf16, int8 x int8, int8-compressed and 4-bit
             weights and the post-ops that such layers carry
  mlp        the fused Llama MLP, on device tensors (amx_mlp.MLP), as a whole block with RMSNorm and residual
             (capi.Mlp.run_block), or on pinned host tensors (the call of a program that keeps its activations in host
             memory, as the CPU library's callers do)
  attention  one-token attention over a bf16 key/value cache whose sequences have their own lengths

listed() holds one case for each situation that differs in what bounds it; draw() gives further sizes of the same ranges.
"""
import math

import torch

from mm_amx_b200 import amx_mlp, capi

# stored bits per weight
WEIGHT_BITS = {"bf16": 16, "w8c": 8, "w8t": 8, "w4": 4, "s8": 8}
OUT_DTYPES = {"bf16": (capi.BF16, torch.bfloat16, 2), "f32": (capi.F32, torch.float32, 4), "s8": (capi.S8, torch.int8, 1)}


def listed():
    return [
        # one generated token through a square projection (query / output) with int8 weights: the smallest call, latency
        dict(name="fc_w8_decode_m1", kind="fc", w="w8c", M=1, K=4096, N=4096, post="", out="bf16"),
        # sixteen sequences decoded together, int8 weights with per-channel scales
        dict(name="fc_w8_decode_m16", kind="fc", w="w8c", M=16, K=4096, N=11008, post="", out="bf16"),
        # a few sequences decoded together, 4-bit weights with group scales
        dict(name="fc_w4_decode_m4", kind="fc", w="w4", M=4, K=4096, N=11008, post="", out="bf16"),
        # a short prompt through a 4-bit layer: too many rows for the decode kernels, too few to be bound by arithmetic
        dict(name="fc_w4_prefill_m100", kind="fc", w="w4", M=100, K=4096, N=11008, post="", out="bf16"),
        # a prompt of odd length through an int8-compressed layer with one scale, bias and GeLU
        dict(name="fc_w8_prefill_m705", kind="fc", w="w8t", M=705, K=2560, N=10240, post="bias,gelu", out="bf16"),
        # the plain bf16 Linear with bias and fp32 result of the reference's own benchmark
        dict(name="fc_bf16_m256", kind="fc", w="bf16", M=256, K=4096, N=4096, post="bias", out="f32"),
        # int8 activations and weights, dequantised per channel, bias, requantised to int8 for the next layer
        dict(name="fc_s8_m2048", kind="fc", w="s8", M=2048, K=4096, N=4096, post="bias,quant", out="s8"),
        # one token through a whole MLP block of a Llama-7B: RMSNorm, gate/up, SiLU, down, residual
        dict(name="mlp_7b_block_m1", kind="mlp", how="block", M=1, K=4096, N=11008),
        # a prompt of ordinary length through the Llama-7B MLP
        dict(name="mlp_7b_m256", kind="mlp", how="device", M=256, K=4096, N=11008),
        # a batch of long prompts through the Llama-70B MLP: the largest call, bound by the tensor cores
        dict(name="mlp_70b_m4096", kind="mlp", how="device", M=4096, K=8192, N=28672),
        # a long prompt whose activations live in pinned host memory, in and out
        dict(name="mlp_7b_host_m2048", kind="mlp", how="host", M=2048, K=4096, N=11008),
        # one decoding step of sixteen sequences between a quarter of and the full cache length, eight query heads per kv head
        dict(name="attention_b16_n4096", kind="attention", B=16, H=64, Hkv=8, N=4096, D=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, decode):
    return rng.randint(1, 16) if decode else _log_int(rng, 17, 4096)


def _features(rng, lo, hi, step):
    """a layer width: mostly a multiple of 128 as model widths are, else of `step` only"""
    v = _log_int(rng, lo, hi)
    step = 128 if rng.random() < 0.7 else step
    return max(lo, v // step * step)


def draw(rng):
    kind = rng.choice(["fc", "fc", "fc", "fc", "mlp", "mlp", "attention"])
    if kind == "fc":
        decode = rng.random() < 0.5
        w = rng.choice(["bf16", "w8c", "w8t", "w4"] if decode else ["bf16", "w8c", "w8t", "w4", "s8"])
        post = rng.choice(["", "bias", "bias,gelu"])
        out = rng.choice(["bf16", "bf16", "f32"])
        if w == "s8" and rng.random() < 0.7:
            post, out = rng.choice(["bias,quant", "bias,gelu,quant"]), "s8"
        # rows are 16-byte aligned in any case; a width need not be a multiple of any tile
        K = _features(rng, 1024, 11008, 32)
        N = _features(rng, 1024, 28672, 8)
        return dict(kind="fc", w=w, M=_rows(rng, decode), K=K, N=N, post=post, out=out)
    if kind == "mlp":
        how = rng.choice(["device", "device", "block", "host"])
        K = _features(rng, 1024, 8192, 64)
        N = min(28672, int(K * rng.uniform(2.5, 3.6)) // 32 * 32)
        return dict(kind="mlp", how=how, M=_rows(rng, how != "host" and rng.random() < 0.5), K=K, N=N)
    G = rng.choice([1, 2, 4, 8])
    Hkv = rng.choice([4, 8, 16, 32])
    B, D = _log_int(rng, 1, 32), rng.choice([64, 128, 128])
    # at most 1 GB of cache
    most = (1 << 30) // (B * Hkv * D * 4)
    return dict(kind="attention", B=B, H=G * Hkv, Hkv=Hkv, N=min(most, _log_int(rng, 200, 16384)), D=D)


def _randn(shape, std, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).mul_(std).to(torch.bfloat16)


def _lengths(B, N):
    """tokens of each sequence: evenly spread from a quarter of the cache to all of it"""
    return [N - (N - N // 4) * i // max(1, B - 1) if B > 1 else N for i in range(B)]


def _prepare_fc(c, g):
    M, K, N, w = c["M"], c["K"], c["N"], c["w"]
    steps, bias, scale, deq, q, per_oc = 0, None, None, 1.0, 1.0, None
    if w in ("s8", "w8c"):
        B = torch.randint(-128 if w == "s8" else -127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        scale = torch.rand(N, generator=g, device="cuda") * 0.049 + 0.001 if w == "s8" else torch.rand(N, generator=g, device="cuda") * 0.019 + 0.001
        steps |= capi.STEP_DEQUANT
    else:
        B = _randn((N, K), 0.02, g)
        steps |= 0 if w == "bf16" else capi.STEP_DEQUANT
    if w == "s8":
        A = torch.randint(-128, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
        weight = capi.Weight(B.data_ptr(), capi.S8, K, N, K, True, capi.PACK_PLAIN)
        deq, per_oc = 1.0 / 512, scale       # activation scale; the layer's own scales are per channel
        q = 127.0 / (2.5 * math.sqrt(K) * 5461.0 * deq * 0.0255)   # about one value in a hundred saturates
    else:
        A = _randn((M, K), 1.0, g)
        mode = {"bf16": capi.PACK_PLAIN, "w8c": capi.PACK_INT8_CHANNEL, "w8t": capi.PACK_QUANT_TENSOR, "w4": capi.PACK_INT4_GROUP}[w]
        weight = capi.Weight(B.data_ptr(), capi.S8 if w == "w8c" else capi.BF16, K, N, K * (1 if w == "w8c" else 2), True, mode,
                             scale.data_ptr() if w == "w8c" else None)
    if "bias" in c["post"]:
        bias = torch.randn(N, generator=g, device="cuda")
        steps |= capi.STEP_BIAS
    steps |= capi.STEP_GELU if "gelu" in c["post"] else 0
    steps |= capi.STEP_QUANT if "quant" in c["post"] else 0
    code, dtype, size = OUT_DTYPES[c["out"]]
    C = torch.empty((M, N), dtype=dtype, device="cuda")
    return dict(kind="fc", w=weight, A=A, dtypeA=capi.S8 if w == "s8" else capi.BF16, M=M, K=K, lda=K * A.element_size(), C=C,
                ldc=N * size, code=code, steps=steps, bias=bias, deq=deq, per_oc=per_oc, q=q)


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if c["kind"] == "fc":
        return _prepare_fc(c, g)
    if c["kind"] == "mlp":
        M, K, N = c["M"], c["K"], c["N"]
        x = _randn((M, K), 1.0, g)
        gate, up, down = _randn((N, K), 0.02, g), _randn((N, K), 0.02, g), _randn((K, N), 0.02, g)
        if c["how"] == "block":
            s = dict(kind="block", x=x, mlp=capi.Mlp(gate.data_ptr(), up.data_ptr(), down.data_ptr(), K, N), M=M, K=K,
                     norm=(1.0 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16), out=torch.empty_like(x))
            s["mlp"].reserve(M)
            return s
        mlp = amx_mlp.MLP(gate, up, down)
        if c["how"] == "host":
            x = x.cpu().pin_memory()
            return dict(kind="mlp", mlp=mlp, x=x, out=torch.empty_like(x).pin_memory())
        return dict(kind="mlp", mlp=mlp, x=x, out=torch.empty_like(x))
    B, H, Hkv, N, D = c["B"], c["H"], c["Hkv"], c["N"], c["D"]
    lens = torch.tensor(_lengths(B, N), dtype=torch.int32, device="cuda")[torch.randperm(B, generator=g, device="cuda")].contiguous()
    q = _randn((B, H, D), 1.0, g)
    k, v = _randn((B, Hkv, N, D), 1.0, g), _randn((B, Hkv, N, D), 1.0, g)
    out = torch.empty((B, H, D), dtype=torch.bfloat16, device="cuda")
    desc = capi.Attention(B, H, Hkv, N, D, q.data_ptr(), H * D * 2, D * 2, k.data_ptr(), v.data_ptr(), Hkv * N * D * 2, N * D * 2,
                          D * 2, out.data_ptr(), H * D * 2, D * 2, capi.BF16, lens.data_ptr(), 1.0 / math.sqrt(D))
    return dict(kind="attention", desc=desc, out=out, keep=(q, k, v, lens))


def run(state):
    s = state
    if s["kind"] == "fc":
        ep = capi.make_epilogue(s["C"].data_ptr(), s["ldc"], s["code"], s["steps"], s["bias"].data_ptr() if s["bias"] is not None else None,
                                s["deq"], s["per_oc"].data_ptr() if s["per_oc"] is not None else None, s["q"])
        s["w"].matmul(s["A"].data_ptr(), s["dtypeA"], s["M"], s["K"], s["lda"], ep)
        return s["C"]
    if s["kind"] == "mlp":
        return s["mlp"].forward(s["x"], s["out"])
    if s["kind"] == "block":
        s["mlp"].run_block(s["x"].data_ptr(), s["K"] * 2, s["M"], 1e-5, s["out"].data_ptr(), s["K"] * 2, s["norm"].data_ptr())
        return s["out"]
    capi.decode_attention(s["desc"])
    return s["out"]


def work(case):
    c = case
    if c["kind"] == "fc":
        M, K, N = c["M"], c["K"], c["N"]
        weights = K * N * WEIGHT_BITS[c["w"]] // 8
        scales = {"w8c": 4 * N, "s8": 4 * N, "w4": 4 * N * ((K + capi.INT4_GROUP - 1) // capi.INT4_GROUP)}.get(c["w"], 0)
        bias = 4 * N if "bias" in c["post"] else 0
        return dict(bytes=weights + scales + bias + M * K * (1 if c["w"] == "s8" else 2) + M * N * OUT_DTYPES[c["out"]][2], flops=2 * M * K * N)
    if c["kind"] == "mlp":
        M, K, N = c["M"], c["K"], c["N"]
        return dict(bytes=3 * K * N * 2 + 2 * M * K * 2, flops=6 * M * K * N)
    tokens = sum(_lengths(c["B"], c["N"]))
    return dict(bytes=tokens * c["Hkv"] * c["D"] * 4 + 2 * c["B"] * c["H"] * c["D"] * 2, flops=4 * tokens * c["H"] * c["D"])


def tolerance(case):
    c = case
    if c["kind"] == "fc":
        if c["out"] == "s8":       # exact int32 sums; the fp32 post-ops may round the other way where a value lies on a tie
            return dict(differ=2e-5)
        # 4-bit weights with more than 16 rows: value x group scale is rounded to bf16 on the way into the product
        if c["out"] == "f32" and (c["w"] != "w4" or c["M"] <= 16):
            return dict(rel=1e-5, max=1e-4)
    # against float64: 1.7e-3 (one bf16 rounding of the result) to 2.4e-3 (a rounded intermediate before it), largest 1.05e-2
    return dict(rel=1e-2, max=4e-2)

"""GPU: GEMM with quantised weights widened into tensor memory (gemm_qt.cu), where one tile is not enough, against the CPU oracle.

Two-valued activations and integer weights (4 bits: power-of-two scales), so that every partial sum is exact in fp32 and the result must
equal the oracle bit for bit; the oracle computes a choice of rows.  Small shapes are in test_gpu_wave.py.
"""
import numpy as np
import pytest

import helpers as H
from mm_amx_b200 import capi
from oracle import port

pytestmark = pytest.mark.gpu

SHAPES = [
    (17, 136, 37000),       # more row blocks than SMs, K that ends inside a piece
    (65, 1024, 20008),      # two rounds of pairs, ragged last row block
    (385, 200, 24000),      # several rounds, two accumulators in turn
    (3000, 520, 2600),      # (one wave of tiles of gemm_wave.cu, as the next)
    (4100, 264, 1032),
    (3000, 3208, 5100),     # token tiles with a ragged last one
    (4100, 4424, 3080),     # ... with the widest tiles: one accumulator
    (520, 8192, 12800),     # K summed in parts, tiles of more than 128 tokens
    (200, 5000, 640),       # parts of K in a cluster, each in several chains (int8; 4 bits: gemm_wave.cu)
]
# calls of SHAPES that gemm_qt.cu takes on 148 SMs
HERE = {"int8": [SHAPES[i] for i in (0, 1, 2, 5, 6, 7, 8)], "int4": [SHAPES[i] for i in (0, 1, 2, 5, 6, 7)]}


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("kind", ["int8", "int4"])
def test_exact(kind, M, K, N):
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    rows = np.unique(np.concatenate([[0, 15, 16, M - 1], rng.integers(0, M, 10)]))
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-7, 8, (N, K), dtype=np.int8)
    if kind == "int8":
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
        acc = port.gemm_bf16_w8(x[rows], B, transposeB=True)
    else:
        B[:, ::128] = 7                     # every group reaches the full range: the scale is 2^-6 exactly
        W = H.bf16_bits(B.astype(np.float32) * np.float32(2.0 ** -6))
        w = H.pack(W, True, capi.PACK_INT4_GROUP)
        acc = port.gemm_bf16(x[rows], W, transposeB=True)
    bias = rng.integers(-8, 9, N).astype(np.float32)
    capi.last_wave_tile()
    before = capi.launch_count()
    assert np.array_equal(H.run_matmul(w, x, capi.F32, steps=capi.STEP_DEQUANT)[rows], acc)
    if H.sms() == 148:
        assert (capi.last_wave_tile() is None and capi.launch_count() - before == 1) == ((M, K, N) in HERE[kind])
    got = H.run_matmul(w, x, capi.BF16, steps=capi.STEP_DEQUANT | capi.STEP_BIAS, bias=bias)[rows]
    assert np.array_equal(got, port.postops(acc, port.BIAS, port.BF16, bias=bias))
    got = H.run_matmul(w, x, capi.S8, steps=capi.STEP_DEQUANT | capi.STEP_BIAS | capi.STEP_QUANT, bias=bias, q_scale=0.5)[rows]
    assert np.array_equal(got, port.postops(acc, port.BIAS | port.QUANT, port.S8, bias=bias, q_scale=0.5))


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("M,K,N", [(40, 520, 392), (65, 1024, 20008), (520, 8192, 12800)])      # one tile, several rounds, parts of K
def test_post_ops_exact(kind, M, K, N):
    """every post-op, scales per column (powers of two, so that all values in front of GeLU are exact)"""
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    rows = np.unique(np.concatenate([[0, 15, 16, M - 1], rng.integers(0, M, 6)]))
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-7, 8, (N, K), dtype=np.int8)
    bias = (rng.integers(-64, 65, N) / 32).astype(np.float32)
    if kind == "int8":
        scales = (2.0 ** -rng.integers(4, 8, N)).astype(np.float32)
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=scales)
        acc = port.gemm_bf16_w8(x[rows], B, transposeB=True) * scales
    else:
        B[:, ::128] = 7
        W = H.bf16_bits(B.astype(np.float32) * np.float32(2.0 ** -6))
        w = H.pack(W, True, capi.PACK_INT4_GROUP)
        acc = port.gemm_bf16(x[rows], W, transposeB=True)
    q = (2.0 ** rng.integers(1, 6, N)).astype(np.float32)
    capi.last_wave_tile()
    for steps, out, kw in [
        (capi.STEP_BIAS | capi.STEP_GELU, capi.BF16, dict(bias=bias)),
        (capi.STEP_GELU, capi.BF16, dict()),
        (capi.STEP_BIAS | capi.STEP_GELU | capi.STEP_QUANT, capi.S8, dict(bias=bias, q_scale=16.0)),
        (capi.STEP_BIAS | capi.STEP_QUANT, capi.S8, dict(bias=bias, q_scale_per_oc=q)),
        (capi.STEP_BIAS | capi.STEP_GELU | capi.STEP_QUANT, capi.F32 if kind == "int4" else capi.BF16, dict(bias=bias, q_scale_per_oc=q)),
    ]:
        got = H.run_matmul(w, x, out, steps=steps | capi.STEP_DEQUANT, **kw)[rows]
        assert np.array_equal(got, port.postops(acc, steps, H.PORT_OF[out], **kw)), (steps, out)
    if H.sms() == 148:
        assert capi.last_wave_tile() is None


def test_extreme_int8_weights_and_scales():
    """every byte value through the widening, with the largest and the smallest scales and activations that leave the result finite"""
    K, N, M = 256, 128, 40
    B = np.tile(np.arange(-128, 128, dtype=np.int8), (N, 1))
    x = np.zeros((M, K), np.float32)
    x[np.arange(M), np.arange(M) * 6] = 1.0
    for scale, unit in [(2.0 ** 127, 2.0 ** -8), (1.0, 2.0 ** 119), (2.0 ** 60, 2.0 ** -126)]:
        scales = np.full(N, scale, np.float32)
        got = H.run_matmul(H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=scales), H.bf16_bits(x * np.float32(unit)), capi.F32, steps=capi.STEP_DEQUANT)
        assert np.array_equal(got, ((x * np.float32(unit)) @ B.T.astype(np.float32)) * scales)


@pytest.mark.parametrize("kind,M,K,N,blocks", [
    ("int8", 1281, 1024, 13000, True), ("int8", 1279, 1024, 13000, False),      # the line at 1.25 K (one block of widened rows)
    ("int8", 1950, 1024, 17000, True), ("int8", 1940, 1024, 17000, False),      # 1.9 K (two blocks)
    ("int8", 400, 200, 40000, True), ("int8", 399, 200, 40000, False),          # 400 rows
    ("int4", 1540, 2048, 10000, False), ("int4", 2920, 2048, 10000, True),      # three quarters of it
])
def test_many_rows_and_short_k(kind, M, K, N, blocks):
    """either side of the line between gemm_qt.cu (one launch) and blocks of widened weights; exact on both, and a capturing stream, whose
    workspace cannot grow, takes the former always"""
    import torch
    rng = np.random.default_rng(M + N)
    rows = np.concatenate([[0, M - 1], rng.integers(0, M, 6)])
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-7, 8, (N, K), dtype=np.int8)
    if kind == "int8":
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
        want = port.gemm_bf16_w8(x[rows], B, transposeB=True)
    else:
        B[:, ::128] = 7
        W = H.bf16_bits(B.astype(np.float32) * np.float32(2.0 ** -6))
        w = H.pack(W, True, capi.PACK_INT4_GROUP)
        want = port.gemm_bf16(x[rows], W, transposeB=True)
    dx, out = H.Dev(x), H.Dev(shape=(M, N), dtype=np.float32, fill=0xCD)
    ep = capi.make_epilogue(out.ptr, out.ld, capi.F32, capi.STEP_DEQUANT)

    def launches(stream):
        before = capi.launch_count()
        w.matmul(dx.ptr, capi.BF16, M, K, 2 * K, ep, stream=stream.cuda_stream)
        return capi.launch_count() - before

    assert (launches(torch.cuda.default_stream()) > 1) == blocks
    capi.sync_check()
    assert np.array_equal(out.numpy()[rows], want)
    out.t.zero_()
    torch.cuda.synchronize()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        assert launches(torch.cuda.current_stream()) == 1
    graph.replay()
    capi.sync_check()
    assert np.array_equal(out.numpy()[rows], want)

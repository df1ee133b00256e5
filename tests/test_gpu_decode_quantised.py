"""GPU: decode-shaped calls with quantised weights (gemv_tq.cu) at the edges of their pieces, against the CPU oracle.

Inputs on which every partial sum is exact in fp32 (two-valued activations; integer weights with unit or power-of-two scales), so
the fp32 result must equal the oracle bit for bit whatever the number of parts K is split into.
"""
import numpy as np
import pytest

import helpers as H
from mm_amx_b200 import capi
from oracle import port

pytestmark = pytest.mark.gpu

SHAPES = [
    (64, 8),          # less than one stage of K, fewer columns than a row block
    (136, 130),       # a K tail in the second stage (int8) / the second group (4 bits); a second row block of two columns
    (4096, 300),      # K in eight parts
    (1000, 4096),     # odd K in eight parts
    (2048, 20008),    # one part, more row blocks than SMs
    (264, 40000),     # more row blocks than CTAs are resident
    (2048, 4360),     # 35, 49, 72 and 94 row blocks: one more than the clusters of 8, 6, 4 and 3 CTAs that are resident together can
    (2048, 6200),     # be given, so K is cut into one part less (int8: with eight accumulators)
    (2304, 9216),
    (2304, 12032),
]


@pytest.mark.parametrize("M", [1, 9, 16])
@pytest.mark.parametrize("K,N", SHAPES)
@pytest.mark.parametrize("kind", ["int8", "int4"])
def test_exact(kind, K, N, M):
    rng = np.random.default_rng(K + 3 * N + M)
    x = H.two_valued_bf16(rng, (M, K))
    if kind == "int8":
        B = rng.integers(-128, 128, (N, K), dtype=np.int8)
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
        acc = port.gemm_bf16_w8(x, B, transposeB=True)
    else:
        q0 = rng.integers(-7, 8, (N, K)).astype(np.float32)
        q0[:, ::128] = 7                    # every group reaches the full range, so the scale is 2^-6 exactly
        B = H.bf16_bits(q0 * np.float32(2.0 ** -6))
        q, d = port.quantize_weight_int4(B)
        w = H.pack(B, True, capi.PACK_INT4_GROUP)
        acc = port.gemm_bf16_w4(x, q, d)
    assert np.array_equal(H.run_matmul(w, x, capi.F32, steps=capi.STEP_DEQUANT), acc)
    bias = rng.integers(-8, 9, N).astype(np.float32)
    got = H.run_matmul(w, x, capi.S8, steps=capi.STEP_DEQUANT | capi.STEP_BIAS | capi.STEP_QUANT, bias=bias, q_scale=2.0 ** -3)
    assert np.array_equal(got, port.postops(acc, port.BIAS | port.QUANT, port.S8, bias=bias, q_scale=2.0 ** -3))

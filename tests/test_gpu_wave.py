"""GPU: the one-wave GEMM (gemm_wave.cu) at the edges of its tiles, for every weight type, against the CPU oracle.
Quantised weights with up to 512 rows, or with K split, go to gemm_qt.cu from most of SHAPES; test_quantised_weights_ragged has shapes that stay.

Inputs on which every partial sum is exact in fp32 (two-valued activations, integer or power-of-two weights), so the result
must equal the oracle bit for bit whatever the tile width, the split of K and the order of summation.
"""
import numpy as np
import pytest

import helpers as H
from mm_amx_b200 import capi
from oracle import port

pytestmark = pytest.mark.gpu

SHAPES = [
    (17, 64, 32),        # one slab of K, one 32-column tile
    (33, 72, 40),        # K and N tails inside one tile
    (17, 8192, 256),     # K split over a whole cluster
    (128, 2080, 1000),   # the last row count of the single-CTA form; a K part that ends inside a stored piece
    (129, 2080, 1000),   # the first one of the pair form, its second CTA nearly without rows
    (100, 4096, 2750),   # several columns tiles, split K, ragged last tile
    (256, 1536, 4104),   # pair form with a split of K
    (300, 200, 9000),    # two row tiles (bf16 and int8 x int8 go to the persistent kernel: 256 x 256 tiles without a split of K)
    (2048, 128, 4096),   # 512-column tiles: all of tensor memory, columns of two MMAs
    (2100, 136, 5000),   # more tiles than one wave: the persistent kernel, with widened blocks for quantised weights (many rows, short K)
]


def check(w, x, acc, steps, bias):
    got = H.run_matmul(w, x, capi.F32, steps=steps)
    assert np.array_equal(got, acc)
    got = H.run_matmul(w, x, capi.BF16, steps=steps | capi.STEP_BIAS, bias=bias)
    assert np.array_equal(got, port.postops(acc, port.BIAS, port.BF16, bias=bias))


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("kind", ["bf16", "s8", "int8_compressed", "int4"])
def test_every_weight_type_exact(kind, M, K, N):
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    bias = rng.integers(-8, 9, N).astype(np.float32)
    if kind == "s8":
        x, B = rng.integers(-128, 128, (M, K), dtype=np.int8), rng.integers(-128, 128, (N, K), dtype=np.int8)
        acc = port.gemm_i8(x, B, transposeB=True)
        w = H.pack(B, True)
        assert np.array_equal(H.run_matmul(w, x, capi.S32), acc)
        q = np.float32(2.0 ** -9)
        got = H.run_matmul(w, x, capi.S8, steps=capi.STEP_BIAS | capi.STEP_QUANT, bias=bias, q_scale=q)
        assert np.array_equal(got, port.postops(acc, port.BIAS | port.QUANT, port.S8, bias=bias, q_scale=q))
        return
    x = H.two_valued_bf16(rng, (M, K))
    if kind == "bf16":
        B = H.two_valued_bf16(rng, (N, K))
        check(H.pack(B, True), x, port.gemm_bf16(x, B, transposeB=True), 0, bias)
    elif kind == "int8_compressed":
        B = rng.integers(-128, 128, (N, K), dtype=np.int8)
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
        check(w, x, port.gemm_bf16_w8(x, B, transposeB=True), capi.STEP_DEQUANT, bias)
    else:
        q0 = rng.integers(-7, 8, (N, K)).astype(np.float32)
        q0[:, ::128] = 7                    # every group reaches the full range, so the scale is 2^-6 exactly
        B = H.bf16_bits(q0 * np.float32(2.0 ** -6))
        q, d = port.quantize_weight_int4(B)
        check(H.pack(B, True, capi.PACK_INT4_GROUP), x, port.gemm_bf16_w4(x, q, d), capi.STEP_DEQUANT, bias)


@pytest.mark.parametrize("M,K,N,n0,n1", [(40, 512, 900, 128, 777), (200, 512, 900, 128, 900), (200, 512, 900, 0, 129)])
def test_column_range_leaves_the_rest_alone(M, K, N, n0, n1):
    rng = np.random.default_rng(M + n1)
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-128, 128, (N, K), dtype=np.int8)
    w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
    got = H.run_matmul(w, x, capi.F32, steps=capi.STEP_DEQUANT, n0=n0, n1=n1)
    assert np.array_equal(got[:, n0:n1], port.gemm_bf16_w8(x, B, transposeB=True)[:, n0:n1])
    rest = np.delete(got, np.s_[n0:n1], axis=1).view(np.uint32)
    assert (rest == 0xCDCDCDCD).all()


@pytest.mark.parametrize("M,K,N", [(200, 4096, 8192), (705, 2560, 10240), (300, 8192, 4096)])
@pytest.mark.parametrize("kind", ["int8_compressed", "int4"])
def test_pair_form_repeats_bit_for_bit(kind, M, K, N):
    """slabs widened by one CTA of a pair are multiplied by the other: every one of 100 launches gives the same bits, with the weights and
    activations out of the caches in every other one"""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    A = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    if kind == "int4":
        B = (torch.randn((N, K), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
        w = capi.Weight(B.data_ptr(), capi.BF16, K, N, 2 * K, True, capi.PACK_INT4_GROUP)
    else:
        B = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        one = torch.ones(N, device="cuda")
        w = capi.Weight(B.data_ptr(), capi.S8, K, N, K, True, capi.PACK_INT8_CHANNEL, one.data_ptr())
    flush = torch.empty(64 << 20, dtype=torch.int32, device="cuda")
    first = None
    for i in range(100):
        C = torch.full((M, N), float("nan"), device="cuda")
        if i & 1:
            flush.fill_(i)
        w.matmul(A.data_ptr(), capi.BF16, M, K, 2 * K, capi.make_epilogue(C.data_ptr(), 4 * N, capi.F32, capi.STEP_DEQUANT))
        first = C if first is None else first
        assert torch.equal(C, first), i
    capi.sync_check()


def test_folded_parts_on_a_capturing_stream():
    """the sums of folded parts need a workspace; a graph owns one of its own, so that a replay does not depend on the stream's, which
    a larger call re-allocates"""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)

    def make(M, K, N):
        A = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
        B = (torch.randn((N, K), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
        w = capi.Weight(B.data_ptr(), capi.BF16, K, N, 2 * K, True, capi.PACK_INT4_GROUP)
        C = torch.zeros((M, N), device="cuda")
        ep = capi.make_epilogue(C.data_ptr(), 4 * N, capi.F32, capi.STEP_DEQUANT)
        return C, lambda stream: w.matmul(A.data_ptr(), capi.BF16, M, K, 2 * K, ep, stream=stream.cuda_stream), (A, w, ep)

    C, call, keep = make(300, 4096, 11008)
    C2, larger, keep2 = make(651, 7680, 12160)
    for warm in (False, True):
        s = torch.cuda.Stream()
        call(torch.cuda.default_stream())
        capi.sync_check()
        assert capi.last_wave_tile()[4] > 1
        want = C.clone()
        torch.cuda.synchronize()
        if warm:
            call(s)
            s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            for _ in range(2):
                call(torch.cuda.current_stream())
        for _ in range(3):
            C.zero_()
            larger(s)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(C, want)
    capi.sync_check()


# kind, M, K, N, tile as capi.last_wave_tile (148 SMs): more than 128 weight rows per CTA, whose columns come from two MMAs
TILES = [
    ("int8", 705, 4096, 7680, (2, 160, 1, 1, 1, 72)),      # halves of 96 and 64 rows
    ("int4", 705, 4096, 7680, (2, 160, 1, 1, 1, 72)),
    ("bf16", 705, 2560, 7680, (2, 160, 1, 1, 1, 72)),
    ("int8", 705, 2560, 10240, (2, 224, 1, 1, 1, 69)),     # 128 and 96 rows; few pieces in the rings
    ("int4", 705, 2560, 10240, (2, 224, 1, 1, 1, 69)),
    ("s8", 705, 2560, 10240, (2, 224, 1, 1, 1, 69)),
    ("int8", 705, 4096, 12288, (2, 256, 1, 1, 1, 72)),     # all of tensor memory, the fewest ring slots
    ("int4", 705, 4096, 12288, (2, 256, 1, 1, 1, 72)),
    ("int8", 35, 6400, 21104, (1, 160, 1, 3, 3, 132)),     # folded parts of K, three accumulators
    ("int8", 256, 4096, 16384, (2, 128, 1, 2, 2, 64)),     # ... in the pair form
    ("int4", 300, 4096, 11008, (2, 160, 1, 1, 3, 70)),     # ... with tiles that leave room for one accumulator
    ("int4", 60, 11008, 16384, (1, 224, 2, 2, 2, 74)),     # ... and two CTAs that share K
]


@pytest.mark.parametrize("kind,M,K,N,tile", TILES)
def test_wide_tiles_exact(kind, M, K, N, tile):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("tiles for 148 SMs")
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    rows = np.unique(np.concatenate([[0, 31, 127, 128, 255, 256, M - 1], rng.integers(0, M, 12)]))      # rows the oracle computes
    rows = rows[rows < M]
    B = rng.integers(-7, 8, (N, K), dtype=np.int8)
    steps = 0
    if kind == "s8":
        x = rng.integers(-128, 128, (M, K), dtype=np.int8)
        w, acc, out = H.pack(B, True), port.gemm_i8(x[rows], B, transposeB=True), capi.S32
    else:
        x, out = H.two_valued_bf16(rng, (M, K)), capi.F32
        if kind == "int8":
            steps = capi.STEP_DEQUANT
            w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
            acc = port.gemm_bf16_w8(x[rows], B, transposeB=True)
        else:
            B[:, ::128] = 7                 # (every group of 4-bit weights reaches the full range: the scale is 2^-6 exactly)
            W = H.bf16_bits(B.astype(np.float32) * np.float32(2.0 ** -6))
            steps = capi.STEP_DEQUANT if kind == "int4" else 0
            w = H.pack(W, True, capi.PACK_INT4_GROUP if kind == "int4" else capi.PACK_PLAIN)
            acc = port.gemm_bf16(x[rows], W, transposeB=True)
    capi.last_wave_tile()
    got = H.run_matmul(w, x, out, steps=steps)
    assert capi.last_wave_tile() == tile
    assert np.array_equal(got[rows], acc)


@pytest.mark.parametrize("M,K,N,n0,n1,tile", [
    (700, 200, 4200, 0, 4200, (2, 96, 1, 1, 1, 66)),       # K that ends inside a stored piece, ragged last tile and column chunk
    (700, 1416, 4200, 0, 4200, (2, 96, 1, 1, 1, 66)),
    (2017, 1408, 4200, 0, 4200, (2, 256, 1, 1, 1, 72)),    # columns of two MMAs
    (700, 1416, 4200, 128, 3977, (2, 96, 1, 1, 1, 63)),    # column ranges
    (700, 520, 5000, 256, 4100, (2, 96, 1, 1, 1, 63)),
])
@pytest.mark.parametrize("kind", ["int8", "int4"])
def test_quantised_weights_ragged(kind, M, K, N, n0, n1, tile):
    if H.sms() != 148:
        pytest.skip("tiles for 148 SMs")
    rng = np.random.default_rng(M + 3 * K + 7 * N + n0)
    rows = np.unique(np.concatenate([[0, 127, 128, 255, 256, M - 1], rng.integers(0, M, 8)]))
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-7, 8, (N, K), dtype=np.int8)
    bias = rng.integers(-8, 9, N).astype(np.float32)
    if kind == "int8":
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
        acc = port.gemm_bf16_w8(x[rows], B, transposeB=True)
    else:
        B[:, ::128] = 7
        W = H.bf16_bits(B.astype(np.float32) * np.float32(2.0 ** -6))
        w = H.pack(W, True, capi.PACK_INT4_GROUP)
        acc = port.gemm_bf16(x[rows], W, transposeB=True)
    for steps, out in ((0, capi.F32), (capi.STEP_BIAS, capi.BF16), (capi.STEP_BIAS | capi.STEP_QUANT, capi.S8)):
        capi.last_wave_tile()
        got = H.run_matmul(w, x, out, steps=steps | capi.STEP_DEQUANT, bias=bias, q_scale=0.5, n0=n0, n1=n1)
        assert capi.last_wave_tile() == tile
        assert np.array_equal(got[rows, n0:n1], port.postops(acc, steps, H.PORT_OF[out], bias=bias, q_scale=0.5)[:, n0:n1])
        assert (np.delete(got, np.s_[n0:n1], axis=1).view(np.uint8) == 0xCD).all()


@pytest.mark.parametrize("sms", [2, 37, 100])
@pytest.mark.parametrize("M,K,N", [(40, 2080, 1000), (200, 4096, 2750), (9, 4096, 3000)])
@pytest.mark.parametrize("kind", ["bf16", "int8_compressed", "int4"])
def test_under_an_sm_limit(kind, M, K, N, sms):
    """fewer SMs change the tile, the split of K and the number of chains, or hand the call to the persistent kernel"""
    capi.set_sm_limit(sms)
    try:
        test_every_weight_type_exact(kind, M, K, N)
    finally:
        capi.set_sm_limit(0)

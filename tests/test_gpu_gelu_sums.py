"""GPU: fp32 results behind GeLU keep the bits that they have always had, whatever split of K other calls take.

The polynomial is ill-conditioned near |x| = 5 in fp32, so another order of the sums in front of it moves outputs by up to 7e-4 of their
rms.  golden/golden_gelu_v1.npz holds a sample of each case's outputs, recorded on a B200 (148 SMs) with the library at commit 3858701:

    PYTHONPATH=. python tests/test_gpu_gelu_sums.py OUT.npz
"""
import os
import sys

import numpy as np
import pytest

import helpers as H
from mm_amx_b200 import capi

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "golden_gelu_v1.npz")

CASES = [
    ("bf16", 4, 5504, 5888),       # decode, 46 row blocks: K in six parts although only five would be resident together
    ("bf16", 6, 4096, 9216),       # decode, 72 row blocks: equal pieces of the whole stream
    ("bf16", 3, 12800, 4096),      # decode, long rows: clusters of eight
    ("bf16", 12, 1280, 1280),      # decode on the tensor cores: one accumulator per piece
    ("bf16", 16, 4096, 4352),
    ("int8", 14, 4768, 9472),      # decode, quantised weights
    ("int8", 1, 2048, 4360),
    ("int4", 5, 2048, 6200),
    ("int8", 54, 1408, 3584),      # prefill that fits one wave of tiles: K split over a cluster
    ("int8", 668, 7360, 1536),
    ("int8", 266, 3072, 23680),    # prefill that does not, K in parts
    ("int8", 1348, 1152, 23040),   # ... in one chain: any path gives these bits
]


def outputs(kind, M, K, N):
    """a sample of the call's results, as bits"""
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    x = H.normal_bf16(rng, (M, K))
    bias = rng.standard_normal(N).astype(np.float32)
    std = 2.5 / np.sqrt(K)              # (pre-activations of a standard deviation of 2.7)
    if kind == "int8":
        B = rng.integers(-127, 128, (N, K), dtype=np.int8)
        w, steps = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.full(N, std / 73.3, np.float32)), capi.STEP_DEQUANT
    else:
        B = H.normal_bf16(rng, (N, K), std)
        w, steps = (H.pack(B, True, capi.PACK_INT4_GROUP), capi.STEP_DEQUANT) if kind == "int4" else (H.pack(B, True), 0)
    got = H.run_matmul(w, x, capi.F32, steps=steps | capi.STEP_BIAS | capi.STEP_GELU, bias=bias)
    return got[rng.integers(0, M, 1024), rng.integers(0, N, 1024)].view(np.uint32)


def name(case):
    return "%s_%d_%d_%d" % case


@pytest.mark.parametrize("case", CASES, ids=name)
def test_bits_are_those_recorded(case):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("recorded with the splits of 148 SMs")
    assert np.array_equal(outputs(*case), np.load(GOLDEN)[name(case)])


def test_captured_calls_give_the_same_bits():
    """blocks of widened weights and their split of K: workspaces of the graph's own, on a fresh stream and where a larger call
    re-allocates the stream's before the replay"""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)

    def make(M, K, N):
        x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
        B = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        scales = torch.full((N,), 2.5 / K ** 0.5 / 73.3, device="cuda")
        w = capi.Weight(B.data_ptr(), capi.S8, K, N, K, True, capi.PACK_INT8_CHANNEL, scales.data_ptr())
        out = torch.zeros((M, N), device="cuda")
        ep = capi.make_epilogue(out.data_ptr(), 4 * N, capi.F32, capi.STEP_DEQUANT | capi.STEP_GELU)
        return out, lambda stream: w.matmul(x.data_ptr(), capi.BF16, M, K, 2 * K, ep, stream=stream.cuda_stream), (x, w, ep)

    out, call, keep = make(266, 3072, 23680)
    out2, larger, keep2 = make(300, 8192, 23680)
    before = capi.launch_count()
    call(torch.cuda.default_stream())
    assert capi.launch_count() - before > 4             # (widened, multiplied in parts of K, added: block by block)
    capi.sync_check()
    want = out.clone()
    torch.cuda.synchronize()
    for warm in (False, True):
        s = torch.cuda.Stream()
        if warm:
            call(s)
            s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            call(torch.cuda.current_stream())
        for _ in range(2):
            out.zero_()
            larger(s)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, want)
    capi.sync_check()


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{name(c): outputs(*c) for c in CASES})

"""GPU: the one-wave GEMM and the one with quantised weights (gemm_qt.cu) sum K in no longer chains than the persistent kernel with its split of
K does for the same call; decode calls with K in fewer parts than places for CTAs allow in no longer ones than with as many.

The tensor core's error grows with the length of a chain of fp32 sums.  Both are run on the same ordinary values (the persistent
kernel in a child process with B200FC_GEMM_WAVE=0) and compared with float64, in fp32 and, behind a bias that cancels the result, in
bf16: there the rounding of the output no longer hides the sums.  4-bit weights have power-of-two scales, so that value x scale is
exact in bf16.  All values are positive, which makes the error proportional to the length of the chains.
"""
import json
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    ("int8", 35, 6400, 21104),    # more chains than accumulators fit beside 160-column tiles
    ("int8", 153, 6496, 4352),    # pair form; the widened blocks have different numbers of chains
    ("int8", 256, 4096, 16384),   # pair form, two accumulators
    ("int4", 202, 7360, 8320),
    ("int4", 300, 4096, 11008),   # tiles that leave room for one accumulator
    ("int4", 651, 7680, 12160),   # ... of 512 columns
    ("int4", 60, 11008, 16384),   # the cluster's parts of K have several chains each
    ("bf16", 256, 4096, 4096),
    # gemm_qt.cu: more than one wave of tiles, K in parts
    ("int8", 442, 4160, 21608),
    ("int8", 571, 10624, 21504),
    ("int4", 519, 3456, 14488),
    # ... one wave, shares of K that no number of parts divides
    ("int8", 60, 8320, 2048),
    ("int8", 28, 3040, 5888),
    ("int4", 19, 4864, 4352),
    ("int4", 33, 10624, 1024),
]

CODE = textwrap.dedent("""
    import json, sys
    import torch
    from mm_amx_b200 import capi
    res = []
    for kind, M, K, N in json.loads(sys.argv[1]):
        g = torch.Generator(device="cuda")
        g.manual_seed(K + N)
        A = torch.randn((M, K), generator=g, device="cuda").abs().to(torch.bfloat16)
        steps = 0 if kind == "bf16" else capi.STEP_DEQUANT
        if kind == "int8":
            B = torch.randint(1, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
            one = torch.ones(N, device="cuda")
            w = capi.Weight(B.data_ptr(), capi.S8, K, N, K, True, capi.PACK_INT8_CHANNEL, one.data_ptr())
        else:
            if kind == "int4":
                B = torch.randint(1, 8, (N, K), generator=g, device="cuda").float()
                B[:, ::128] = 7
                B = (B / 64).to(torch.bfloat16)
            else:
                B = torch.randn((N, K), generator=g, device="cuda").abs().to(torch.bfloat16)
            w = capi.Weight(B.data_ptr(), capi.BF16, K, N, 2 * K, True, capi.PACK_INT4_GROUP if kind == "int4" else capi.PACK_PLAIN)
        def call(A, out, code, steps, bias=None):
            ep = capi.make_epilogue(out.data_ptr(), N * out.element_size(), code, steps, bias.data_ptr() if bias is not None else None)
            w.matmul(A.data_ptr(), capi.BF16, M, K, 2 * K, ep)
            capi.sync_check()
            return out.double()
        ref = torch.cat([A.double() @ B[i:i + 2048].double().t() for i in range(0, N, 2048)], 1)
        c = call(A, torch.empty((M, N), device="cuda"), capi.F32, steps)
        same = A[:1].expand(M, K).contiguous()                  # all rows alike: one bias per column cancels them
        bias = -ref[0].float()
        r = call(same, torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), capi.BF16, steps | capi.STEP_BIAS, bias)
        r -= ref[0] + bias.double()
        res.append([float((c - ref).norm() / ref.norm()), float(r.norm() / (ref[0].norm() * M ** 0.5))])
    print("errors", json.dumps(res))
""")


def errors(**switches):
    env = dict(os.environ, **switches)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env["PYTHONPATH"] = os.pathsep.join([root, env.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", CODE, json.dumps(SHAPES)], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.split("errors", 1)[1])


def test_chains_are_no_longer_than_with_the_split_of_k_subprocess():
    for shape, wave, split in zip(SHAPES, errors(), errors(B200FC_GEMM_WAVE="0")):
        for what, e, bound in zip(("fp32", "bf16"), wave, split):
            # 5 %: the chains end at other slabs of K and are added in another order; one chain fewer of eight is 14 %
            assert e <= 1.05 * bound, (shape, what, e, bound)
            assert bound < 4e-6, (shape, what, bound)           # (that is, the persistent kernel did split K)


# clusters of fewer CTAs than there are places for, with chains of sums cut inside the CTAs (bf16 rows that are not 16-byte aligned, and up to
# eight rows: mma.sync; more: four accumulators; quantised weights: more accumulators or levels of sums)
DECODE = [
    ("bf16", 4, 4096, 4352, 0), ("bf16", 12, 4096, 4352, 2), ("bf16", 12, 4096, 4352, 0), ("bf16", 4, 4096, 9216, 0), ("bf16", 5, 12800, 4096, 0),
    ("int8", 4, 4096, 4352, 0), ("int8", 13, 9216, 6272, 0), ("int8", 4, 4096, 4352, 2), ("int8", 12, 4096, 6272, 2),
    ("int4", 4, 4096, 4352, 0), ("int4", 13, 9216, 6272, 0),
]


@pytest.mark.parametrize("kind,M,K,N,shift", DECODE)
def test_decode_chains_are_no_longer_than_with_every_place_taken(kind, M, K, N, shift):
    """Positive values, so that GeLU is the identity on all results: fp32 behind it keeps the split of K into as many parts as there are
    places (see test_gpu_gelu_sums.py), and its error against float64 is the bound."""
    import torch
    from mm_amx_b200 import capi
    g = torch.Generator(device="cuda")
    g.manual_seed(K + N + M)
    A = torch.randn((M, K), generator=g, device="cuda").abs().to(torch.bfloat16)
    shifted = torch.empty(M * K + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(M, K).copy_(A)
    if kind == "int8":
        B = torch.randint(1, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        one = torch.ones(N, device="cuda")
        w = capi.Weight(B.data_ptr(), capi.S8, K, N, K, True, capi.PACK_INT8_CHANNEL, one.data_ptr())
    else:
        B = torch.randn((N, K), generator=g, device="cuda").abs().to(torch.bfloat16)
        if kind == "int4":
            B = torch.randint(1, 8, (N, K), generator=g, device="cuda").float()
            B[:, ::128] = 7
            B = (B / 64).to(torch.bfloat16)
        w = capi.Weight(B.data_ptr(), capi.BF16, K, N, 2 * K, True, capi.PACK_INT4_GROUP if kind == "int4" else capi.PACK_PLAIN)
    ref = A.double() @ B.double().t()

    def call(steps):
        out = torch.empty((M, N), device="cuda")
        w.matmul(shifted.data_ptr(), capi.BF16, M, K, 2 * K, capi.make_epilogue(out.data_ptr(), 4 * N, capi.F32, steps | (capi.STEP_DEQUANT if kind != "bf16" else 0)))
        capi.sync_check()
        return out

    every, fewer = call(capi.STEP_GELU), call(0)
    assert float(ref.min()) > 6.0 and not torch.equal(every, fewer)
    bound, e = (float((c.double() - ref).norm() / ref.norm()) for c in (every, fewer))
    assert e <= 1.05 * bound, (e, bound)

"""GPU: the persistent GEMMs (gemm_tc.cu), their split of K and the blocks of widened weights in front of them.

Calls whose output fits one wave of tiles go to gemm_wave.cu by default, which takes the shapes that the older tests were written for.
Here those tests run again in child processes (the switches are read once per process) with the one-wave kernel off, and
with the single-CTA kernel forced.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import helpers as H
from mm_amx_b200 import capi
from oracle import port

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("M,K,N,n0,n1", [
    (130, 8192, 4400, 0, 4400),       # three blocks of 2048 rows, the last of 304 columns
    (64, 8192, 4400, 2176, 4400),     # starts inside the second block
])
def test_column_range_over_widened_blocks(kind, M, K, N, n0, n1):
    """as one wave by default; with B200FC_GEMM_WAVE=0 (below) block by block, each with its part of C, bias and scales"""
    rng = np.random.default_rng(M + n0)
    x = H.normal_bf16(rng, (M, K))
    bias = rng.standard_normal(N).astype(np.float32)
    if kind == "int8":
        B = rng.integers(-127, 128, (N, K), dtype=np.int8)
        scale = rng.uniform(0.001, 0.02, N).astype(np.float32)
        w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=scale)
        ref = port.gemm_bf16_w8(x, B, transposeB=True) * scale + bias
    else:
        W = H.normal_bf16(rng, (N, K), 0.02)
        q, d = port.quantize_weight_int4(W)
        w = H.pack(W, True, capi.PACK_INT4_GROUP)
        ref = port.gemm_bf16(x, H.bf16_bits(port.dequant_int4(q, d)), transposeB=True) + bias
    got = H.run_matmul(w, x, capi.F32, steps=capi.STEP_DEQUANT | capi.STEP_BIAS, bias=bias, n0=n0, n1=n1)
    assert H.rel_to_max(got[:, n0:n1], ref[:, n0:n1]) < 1e-5
    rest = np.delete(got, np.s_[n0:n1], axis=1).view(np.uint32)
    assert (rest == 0xCDCDCDCD).all()


AGAIN = {
    "B200FC_GEMM_WAVE=0": [
        "test_gpu_fc.py::test_compressed_weights_prefill_blocks", "test_gpu_fc.py::test_split_k_shapes_exact",
        "test_gpu_fc.py::test_many_tiles_exact", "test_gpu_int4.py::test_int4_prefill_blocks", "test_gpu_mlp.py::test_mlp_long_k_few_tiles",
        "test_gpu_wave.py::test_every_weight_type_exact", "test_gpu_wave.py::test_column_range_leaves_the_rest_alone",
        "test_gpu_persistent.py::test_column_range_over_widened_blocks"],
    "B200FC_GEMM_CTAS=1": ["test_gpu_fc.py::test_many_tiles_exact", "test_gpu_wave.py::test_every_weight_type_exact"],
}


@pytest.mark.parametrize("switch", sorted(AGAIN))
def test_again_without_the_one_wave_kernel_subprocess(switch):
    env = dict(os.environ, **dict([switch.split("=")]))
    ids = [os.path.join(HERE, t) for t in AGAIN[switch]]
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"] + ids, env=env, cwd=os.path.dirname(HERE),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and " passed" in r.stdout and "skipped" not in r.stdout, r.stdout[-4000:] + r.stderr[-2000:]

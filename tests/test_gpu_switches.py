"""GPU: the environment switches that force a kernel reach it for every size, also where another kernel is the default.

Each is read once per process, hence the child processes; what ran is told apart by the number of launches, and the result
must equal the CPU oracle bit for bit (two-valued activations, integer weights).
"""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

CODE = textwrap.dedent("""
    import sys
    import numpy as np
    import helpers as H
    from mm_amx_b200 import capi
    from oracle import port
    M, K, N, launches = map(int, sys.argv[1:])
    rng = np.random.default_rng(M + K + N)
    x = H.two_valued_bf16(rng, (M, K))
    B = rng.integers(-128, 128, (N, K), dtype=np.int8)
    w = H.pack(B, True, capi.PACK_INT8_CHANNEL, scales=np.ones(N, np.float32))
    before = capi.launch_count()
    got = H.run_matmul(w, x, capi.F32, steps=capi.STEP_DEQUANT)
    assert capi.launch_count() - before == launches, capi.launch_count() - before
    assert np.array_equal(got, port.gemm_bf16_w8(x, B, transposeB=True))
    print("switch ok")
""")


@pytest.mark.parametrize("switch,M,K,N,launches", [
    ("", 64, 8192, 2600, 1),                        # one-wave kernel
    ("B200FC_GEMM_WAVE=0", 64, 8192, 2600, 6),      # two widened blocks, each multiplied with a split of K and reduced
    ("B200FC_GEMM_CTAS=1", 64, 8192, 2600, 4),      # ... without that split
    ("B200FC_GEMM_CTAS=2", 64, 8192, 2600, 6),
    ("", 5, 4096, 1024, 1),                         # tensor-core decode kernel
    ("B200FC_GEMV_XIMG=1", 5, 4096, 1024, 2),       # activations converted by a launch of their own
    ("B200FC_GEMV_XIMG=0", 5, 4096, 1024, 1),
    ("B200FC_GEMV_STREAMK=1", 16, 4096, 11008, 2),  # (pieces of more than two chunks: converted activations by default)
])
def test_switch_subprocess(switch, M, K, N, launches):
    env = dict(os.environ, **dict([switch.split("=")] if switch else []))
    here = os.path.dirname(os.path.abspath(__file__))
    env["PYTHONPATH"] = os.pathsep.join([here, os.path.dirname(here), env.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", CODE] + [str(v) for v in (M, K, N, launches)], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and "switch ok" in r.stdout, r.stdout + r.stderr

"""CPU: chains of sums that gemm_qt.cu cuts K into (csrc/split_k.h), with the kernel's own arithmetic for a CTA's share and its parts."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "split_k.h"
int main() {
    int bad = 0;
    for (int stages = 1; stages <= 200; stages++)
        for (int S = 1; S <= 8 && S <= stages; S++)
            for (int chains = 1; chains <= 24; chains++)
                for (int even = 0; even < 2; even++) {
                    const int given = b200fc::parts_of_share(stages, S, chains, even);
                    int total = 0, longest = 0, several = 0;
                    for (int split = 0; split < S; split++) {
                        const int n = stages * (split + 1) / S - stages * split / S, parts = std::min(given, n);
                        total += parts;
                        several |= parts > 1;
                        for (int q = 0; q < parts; q++) longest = std::max(longest, n * (q + 1) / parts - n * q / parts);
                    }
                    const bool enough = total >= std::min(chains, stages);
                    const bool short_ones = !even || !several || longest <= std::max(1, stages / chains);
                    if (!enough || !short_ones) { if (bad++ < 10) std::printf("stages %d S %d chains %d even %d: %d chains, longest %d\n", stages, S, chains, even, total, longest); }
                }
    return bad != 0;
}
"""


def test_chains_of_sums(tmp_path):
    src, exe = tmp_path / "split.cpp", str(tmp_path / "split")
    src.write_text(PROGRAM)
    subprocess.check_call(["/usr/bin/g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "mm_amx_b200", "csrc"), str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

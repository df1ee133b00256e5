"""CPU: which host buffers the kernels of the host-buffer MLP call may touch (csrc/host_span.h), with made-up answers of the driver."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "host_span.h"
using namespace b200fc;
// pinned registrations of a process: [0x10000, +0x8000), [0x20000, +0x8000) with a hole between them, [0x28000, +0x1000) right behind,
// read-only [0x40000, +0x1000), and one whose device address differs, [0x50000, +0x1000) at 0x90000
static bool query(const void* p, HostRange* r) {
    const uintptr_t a = (uintptr_t)p;
    struct { uintptr_t host, dev; size_t size; bool w; } t[] = {
        {0x10000, 0x10000, 0x8000, true}, {0x20000, 0x20000, 0x8000, true}, {0x28000, 0x28000, 0x1000, true},
        {0x40000, 0x40000, 0x1000, false}, {0x50000, 0x90000, 0x1000, true}};
    for (auto& e : t)
        if (a >= e.host && a < e.host + e.size) { *r = HostRange{true, true, e.w, a - e.host + e.dev, e.dev, e.size}; return true; }
    return false;
}
static int bad;
static void expect(uintptr_t p, int64_t ld, size_t bytes, bool write, uintptr_t want) {
    const uintptr_t got = span_on_device((const void*)p, ld, bytes, write, query);
    if (got != want) { std::printf("%zx + %zx ld %lld: %zx, not %zx\n", (size_t)p, bytes, (long long)ld, (size_t)got, (size_t)want); bad = 1; }
}
int main() {
    expect(0x10000, 64, 0x8000, true, 0x10000);      // all of a registration, and parts of it
    expect(0x10010, 64, 0x7ff0, true, 0x10010);
    expect(0x17ff0, 64, 16, true, 0x17ff0);
    expect(0x10000, 64, 0x8001, true, 0);            // past its end
    expect(0x10000, 0x10000, 0x10040, true, 0);      // first and last row in two registrations, a hole between them
    expect(0x20000, 64, 0x9000, true, 0);            // two registrations without a hole: not known to stay together
    expect(0x18000, 64, 64, true, 0);                // not pinned
    expect(0x10008, 64, 64, true, 0);                // rows that are not 16-byte aligned
    expect(0x10000, 72, 64, true, 0);
    expect(0x10000, 64, 0, true, 0);
    expect(0x40000, 64, 0x1000, false, 0x40000);     // read-only memory
    expect(0x40000, 64, 0x1000, true, 0);
    expect(0x50010, 64, 0xff0, true, 0x90010);       // another address on the device
    expect(0x50010, 64, 0x1000, true, 0);
    auto managed = [](const void* p, HostRange* r) { query(p, r); r->pinned = false; return true; };
    if (span_on_device((const void*)0x10000, 64, 64, false, managed)) bad = 1;
    return bad;
}
"""


def test_choice_of_path(tmp_path):
    src, exe = tmp_path / "span.cpp", str(tmp_path / "span")
    src.write_text(PROGRAM)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "mm_amx_b200", "csrc"), str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
